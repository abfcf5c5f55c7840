// Vertex-triangle narrow phase and non-penetration projection
// (framework/physics/collision_constraints_x.py __vt_st / __vt_dy / __tv_st,
// framework/collision/distance.py d_type_PT, d_PP/d_PE/d_PT and gradients),
// followed by update_dx (XPBD.py:384-387).
//
// Corrections are accumulated in 64-bit fixed point (40 fractional bits) with
// integer atomics, so the sum does not depend on the order in which threads
// arrive (the reference uses float atomics, whose result does).
#include "sx_common.cuh"
#include "sx_exact.cuh"
#include "sx_sweep.cuh"

namespace sx {

// Reciprocals and quotients of the narrow phase, two bodies with the same
// value: IEEE = false is straight-line code (sx_exact.cuh) that records the
// operands' magnitudes; when they leave [2^-100, 2^100] (degenerate triangles,
// coincident points) the caller evaluates the pair again with '/'.  The three
// 2x2 solves of a classification then run side by side: a pair's chain of
// dependent divisions, not the chip's throughput, is what a contact sweep over
// a few thousand pairs waits for.
template <bool IEEE>
struct Arith {
    float lo = 1.0f, hi = 1.0f;
    __device__ __forceinline__ void note(float v) {
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
    }
    __device__ __forceinline__ float rcp(float b) {
        if (IEEE) return 1.0f / b;
        note(fabsf(b));
        return rcp_rn(b);
    }
    __device__ __forceinline__ float div(float a, float b) {
        if (IEEE) return a / b;
        const float q = div_rn(a, b, rcp(b));
        note(a == 0.0f ? 1.0f : fabsf(a));
        note(a == 0.0f ? 1.0f : fabsf(q));
        return q;
    }
    // min and max pass over a NaN: both bodies then give NaN
    __device__ __forceinline__ bool ok() const {
        return IEEE || (lo >= 7.88860905e-31f && hi <= 1.26765060e30f);  // 2^-100, 2^100
    }
};

// 2x2 solve A^{-1} b with A^{-1} = (1/det) [[a11, -a01], [-a10, a00]]
template <typename A>
__device__ __forceinline__ void solve2(A& ar, float a00, float a01, float a10, float a11, float b0, float b1,
                                       float* p0, float* p1) {
    float det = a00 * a11 - a01 * a10;
    float id = ar.rcp(det);
    float m00 = id * a11, m01 = id * (-a01), m10 = id * (-a10), m11 = id * a00;
    *p0 = m00 * b0 + m01 * b1;
    *p1 = m10 * b0 + m11 * b1;
}

// distance.py:5-47
template <typename A>
__device__ __forceinline__ int d_type_PT(A& ar, V3 v0, V3 v1, V3 v2, V3 v3) {
    const V3 v12 = sub(v2, v1), v13 = sub(v3, v1);
    const V3 n = cross(v12, v13);
    const V3 v13n = cross(v12, n);
    const V3 v10 = sub(v0, v1);
    const V3 v32 = sub(v3, v2), v32n = cross(v32, n), v20 = sub(v0, v2);
    const V3 v31 = sub(v1, v3), v31n = cross(v31, n), v30 = sub(v0, v3);
    float p00, p01, p10, p11, p20, p21;
    solve2(ar, dot(v12, v12), dot(v12, v13n), dot(v13n, v12), dot(v13n, v13n), dot(v12, v10), dot(v13n, v10), &p00,
           &p01);
    solve2(ar, dot(v32, v32), dot(v32, v32n), dot(v32n, v32), dot(v32n, v32n), dot(v32, v20), dot(v32n, v20), &p10,
           &p11);
    solve2(ar, dot(v31, v31), dot(v31, v31n), dot(v31n, v31), dot(v31n, v31n), dot(v31, v30), dot(v31n, v30), &p20,
           &p21);
    int dt = 6;
    if (p20 <= 0.0f && p10 >= 1.0f) dt = 2;
    if (p10 <= 0.0f && p00 >= 1.0f) dt = 1;
    if (p00 <= 0.0f && p20 >= 1.0f) dt = 0;
    if (p20 > 0.0f && p20 < 1.0f && p21 >= 0.0f) dt = 5;
    if (p10 > 0.0f && p10 < 1.0f && p11 >= 0.0f) dt = 4;
    if (p00 > 0.0f && p00 < 1.0f && p01 >= 0.0f) dt = 3;
    return dt;
}

__device__ __forceinline__ float d_PP(V3 a, V3 b) {
    V3 d = sub(a, b);
    return dot(d, d);
}
template <typename A>
__device__ __forceinline__ float d_PE(A& ar, V3 p, V3 e0, V3 e1) {
    V3 c = cross(sub(e0, p), sub(e1, p));
    V3 e = sub(e1, e0);
    return ar.div(dot(c, c), dot(e, e));
}
template <typename A>
__device__ __forceinline__ float d_PT(A& ar, V3 p, V3 t0, V3 t1, V3 t2) {
    V3 b = cross(sub(t1, t0), sub(t2, t0));
    float s = dot(sub(p, t0), b);
    return ar.div(s * s, dot(b, b));
}
// Closed-form gradients of the squared distances:
//  PP: g_a = 2(a-b), g_b = -g_a
//  PE: c=(e0-p)x(e1-p), L=|e1-e0|^2, d=c.c/L;
//      g_e0 = (2 (e1-p)xc + 2d (e1-e0))/L, g_e1 = (2 cx(e0-p) - 2d (e1-e0))/L,
//      g_p = -(g_e0 + g_e1)
//  PT: n=(t1-t0)x(t2-t0), r=p-t0, s=r.n, N=n.n, d=s^2/N;
//      g_p = 2sn/N, g_t1 = (2s (t2-t0)xr - 2d (t2-t0)xn)/N,
//      g_t2 = (2s rx(t1-t0) - 2d nx(t1-t0))/N, g_t0 = -(g_p + g_t1 + g_t2)
__device__ __forceinline__ void g_PP(V3 a, V3 b, V3* ga, V3* gb) {
    *ga = scale(2.0f, sub(a, b));
    *gb = neg(*ga);
}
template <typename A>
__device__ __forceinline__ void g_PE(A& ar, V3 p, V3 e0, V3 e1, V3* gp, V3* g0, V3* g1) {
    V3 a = sub(e0, p), b = sub(e1, p);
    V3 c = cross(a, b);
    V3 e = sub(e1, e0);
    float L = dot(e, e);
    float iL = ar.rcp(L);
    float d = dot(c, c) * iL;
    V3 bc = cross(b, c), ca = cross(c, a);
    float td = 2.0f * d;
    V3 t0 = add(scale(2.0f, bc), scale(td, e));
    V3 t1 = sub(scale(2.0f, ca), scale(td, e));
    *g0 = scale(iL, t0);
    *g1 = scale(iL, t1);
    *gp = neg(add(*g0, *g1));
}
template <typename A>
__device__ __forceinline__ void g_PT(A& ar, V3 p, V3 t0, V3 t1, V3 t2, V3* gp, V3* g0, V3* g1, V3* g2) {
    V3 u = sub(t1, t0), w = sub(t2, t0);
    V3 n = cross(u, w);
    V3 r = sub(p, t0);
    float s = dot(r, n);
    float N = dot(n, n);
    float iN = ar.rcp(N);
    float d = (s * s) * iN;
    float ts = 2.0f * s, td = 2.0f * d;
    *gp = scale(ts * iN, n);
    V3 a1 = sub(scale(ts, cross(w, r)), scale(td, cross(w, n)));
    V3 a2 = sub(scale(ts, cross(r, u)), scale(td, cross(n, u)));
    *g1 = scale(iN, a1);
    *g2 = scale(iN, a2);
    *g0 = neg(add(add(*gp, *g1), *g2));
}

__device__ __forceinline__ int region_mask(int dtype) {
    // bit k set: vertex k (0 = query point, 1..3 = triangle) takes part
    return dtype == 0 ? 0x3 : dtype == 1 ? 0x5 : dtype == 2 ? 0x9 : dtype == 3 ? 0x7 : dtype == 4 ? 0xD
         : dtype == 5 ? 0xB : dtype == 6 ? 0xF : 0;
}

// The feature of region dt: triangle corner a of a vertex region, the edge
// (a, b) of an edge region, so that a warp whose pairs lie in several regions
// runs the point, edge and face code once each, not once per region.
__device__ __forceinline__ V3 region_a(int dt, const V3 x[4]) {
    return dt == 0 || dt == 3 || dt == 5 ? x[1] : dt == 1 || dt == 4 ? x[2] : x[3];
}
__device__ __forceinline__ V3 region_b(int dt, const V3 x[4]) { return dt == 3 ? x[2] : x[3]; }

template <typename A>
__device__ __forceinline__ float pt_distance(A& ar, int dt, const V3 x[4]) {
    if (dt == 6) return d_PT(ar, x[0], x[1], x[2], x[3]);
    if (dt <= 2) return d_PP(x[0], region_a(dt, x));
    return d_PE(ar, x[0], region_a(dt, x), region_b(dt, x));
}
// zero for the vertices that do not take part
template <typename A>
__device__ __forceinline__ void pt_gradient(A& ar, int dt, const V3 x[4], V3 g[4]) {
    if (dt == 6) {
        g_PT(ar, x[0], x[1], x[2], x[3], &g[0], &g[1], &g[2], &g[3]);
        return;
    }
    const V3 zero{0.0f, 0.0f, 0.0f};
    V3 ga, gb = zero;
    if (dt <= 2)
        g_PP(x[0], region_a(dt, x), &g[0], &ga);
    else
        g_PE(ar, x[0], region_a(dt, x), region_b(dt, x), &g[0], &ga, &gb);
    g[1] = dt == 0 || dt == 3 || dt == 5 ? ga : zero;
    g[2] = dt == 1 || dt == 4 ? ga : dt == 3 ? gb : zero;
    g[3] = dt == 2 ? ga : dt == 4 || dt == 5 ? gb : zero;
}

// One candidate: its region, squared distance and, where d < dHat, gradients,
// schur complement and multiplier of its kind.
//   VT_ST (collision_constraints_x.py:6-69): dynamic vertex vs static triangle;
//     w[0] = m_inv, schur = w0 g0.g0, ld = c (dHat - d) / (c schur + 1)
//   VT_DY (:176-310): self contact; w[k] = fixed m_inv, schur = the sum of
//     w_k g_k.g_k over the region's vertices + 1e-4, ld = (dHat - d) / schur
//   TV_ST (:72-173): static vertex vs dynamic triangle; as VT_ST with the sum
//     over the triangle's vertices
// The kind is a run-time value: one copy of the classification serves a warp
// whose lanes hold different kinds, and fits the instruction cache.
enum PairKind { VT_ST, VT_DY, TV_ST };
struct PairSolve {
    int dt;
    float d, schur, ld;
    V3 g[4];
};
// the vertices a kind corrects, among those of the region
__device__ __forceinline__ int moved_mask(int kind, int dt) {
    return region_mask(dt) & (kind == VT_ST ? 0x1 : kind == TV_ST ? 0xE : 0xF);
}
template <typename A>
__device__ __forceinline__ void pair_classify(A& ar, const V3 x[4], PairSolve& r) {
    r.dt = d_type_PT(ar, x[0], x[1], x[2], x[3]);
    r.d = pt_distance(ar, r.dt, x);
}
// gradients, schur complement and multiplier of a pair in contact
template <typename A>
__device__ __forceinline__ void pair_correction(A& ar, int kind, const V3 x[4], const float w[4], float dHat,
                                                float compliance, PairSolve& r) {
    pt_gradient(ar, r.dt, x, r.g);
    const int m = moved_mask(kind, r.dt);
    float s = 0.0f;
    bool first = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float t = w[k] * dot(r.g[k], r.g[k]);
        if (m & (1 << k)) {
            s = first ? t : s + t;
            first = false;
        }
    }
    const float gap = dHat - r.d;
    if (kind == VT_DY) s = s + 1e-4f;
    r.ld = ar.div(kind == VT_DY ? gap : compliance * gap, kind == VT_DY ? s : compliance * s + 1.0f);
    r.schur = s;
}
template <bool IEEE>
__device__ __forceinline__ bool pair_solve(int kind, const V3 x[4], const float w[4], float dHat, float compliance,
                                           PairSolve& r) {
    Arith<IEEE> ar;
    pair_classify(ar, x, r);
    r.schur = r.ld = 0.0f;
    if (r.d < dHat) pair_correction(ar, kind, x, w, dHat, compliance, r);
    return ar.ok();
}

__device__ __forceinline__ void acc_add(long long* dx, int* nc, int v, float a, V3 g, int* bad) {
    long long c0 = to_fix(a * g.x, bad), c1 = to_fix(a * g.y, bad), c2 = to_fix(a * g.z, bad);
    atomicAdd((unsigned long long*)(dx + 3 * v), (unsigned long long)c0);
    atomicAdd((unsigned long long*)(dx + 3 * v + 1), (unsigned long long)c1);
    atomicAdd((unsigned long long*)(dx + 3 * v + 2), (unsigned long long)c2);
    atomicAdd(nc + v, 1);
}

struct PairOut {
    int* pair;
    float* g;
    float* schur;
    int* num;
    int cap;
    __device__ __forceinline__ void rec(size_t q, int& cnt, int face, int dtype, const V3 gg[4], float s) {
        if (!num || cnt >= cap) return;
        size_t o = q * cap + cnt;
        pair[2 * o] = face;
        pair[2 * o + 1] = dtype;
        float4* g4 = reinterpret_cast<float4*>(g) + 4 * o;
        for (int k = 0; k < 4; ++k) g4[k] = make_float4(gg[k].x, gg[k].y, gg[k].z, 0.0f);
        schur[o] = s;
        ++cnt;
    }
};

// The corrections of one candidate in contact.  mi: m_inv, w: the kind's weights.
__device__ __forceinline__ void pair_apply(int kind, const int vv[4], const float mi[4], const float w[4],
                                           const PairSolve& r, long long* dx, int* nc, int* bad) {
    const int m = moved_mask(kind, r.dt);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!(m & (1 << k))) continue;
        // region 0 of VT_DY applies m_inv without `fixed` (collision_constraints_x.py:199-200)
        acc_add(dx, nc, vv[k], (kind == VT_DY && r.dt == 0 ? mi[k] : w[k]) * r.ld, r.g[k], bad);
    }
}

// Weights of a candidate: VT_ST has no `fixed` factor (collision_constraints_x.py:58);
// vertices of the static mesh have none.
__device__ __forceinline__ void pair_weights(int kind, const int vv[4], const float* __restrict__ fixed,
                                             const float* __restrict__ m_inv, float mi[4], float w[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const bool dyn = kind == VT_DY || (k == 0) == (kind == VT_ST);
        mi[k] = dyn ? m_inv[vv[k]] : 0.0f;
        w[k] = !dyn ? 0.0f : kind == VT_ST ? mi[k] : fixed[vv[k]] * mi[k];
    }
}

// The same candidate with the compiler's divisions, out of line: rare.
__device__ __noinline__ int pair_project_ieee(int kind, int4 v, V3 x0, V3 x1, V3 x2, V3 x3,
                                              const float* __restrict__ fixed, const float* __restrict__ m_inv,
                                              float dHat, float compliance, long long* dx, int* nc) {
    const int vv[4] = {v.x, v.y, v.z, v.w};
    const V3 x[4] = {x0, x1, x2, x3};
    float mi[4], w[4];
    pair_weights(kind, vv, fixed, m_inv, mi, w);
    PairSolve r;
    int bad = 0;
    pair_solve<true>(kind, x, w, dHat, compliance, r);
    if (r.d < dHat) pair_apply(kind, vv, mi, w, r, dx, nc, &bad);
    return bad;
}

// One candidate's corrections (__vt_st, __vt_dy or __tv_st); the weights are
// loaded before the classification, which hides their latency.
__device__ __forceinline__ void pair_project(int kind, int4 v, const V3 x[4], const float* __restrict__ fixed,
                                             const float* __restrict__ m_inv, float dHat, float compliance,
                                             long long* dx, int* nc, int* bad) {
    const int vv[4] = {v.x, v.y, v.z, v.w};
    float mi[4], w[4];
    pair_weights(kind, vv, fixed, m_inv, mi, w);
    PairSolve r;
    if (!pair_solve<false>(kind, x, w, dHat, compliance, r))
        *bad |= pair_project_ieee(kind, v, x[0], x[1], x[2], x[3], fixed, m_inv, dHat, compliance, dx, nc);
    else if (r.d < dHat)
        pair_apply(kind, vv, mi, w, r, dx, nc, bad);
}

// The same for kernels that are short of registers: without a call, the weights and
// gradients (with '/', which takes fewer) only of a pair in contact.  In the
// persistent substep, 64 registers a thread, pair_project spills and its call keeps
// registers from the sweep: frames of 512 / 64 falling cloths in fast arithmetic 24.1 /
// 4.9 ms with it, 23.1 / 4.6 with this (23.3 / 4.6 with no projection in the kernel),
// of 512 lying on their boxes 57.9 and 50.5.
__device__ __forceinline__ void pair_project_lean(int kind, int4 v, const V3 x[4], const float* __restrict__ fixed,
                                                  const float* __restrict__ m_inv, float dHat, float compliance,
                                                  long long* dx, int* nc, int* bad) {
    PairSolve r;
    Arith<false> ar;
    Arith<true> ieee;
    pair_classify(ar, x, r);
    if (!ar.ok()) pair_classify(ieee, x, r);
    if (!(r.d < dHat)) return;
    const int vv[4] = {v.x, v.y, v.z, v.w};
    float mi[4], w[4];
    pair_weights(kind, vv, fixed, m_inv, mi, w);
    pair_correction(ieee, kind, x, w, dHat, compliance, r);
    pair_apply(kind, vv, mi, w, r, dx, nc, bad);
}

// The same, for the walk that records its pairs: r also receives the region,
// the gradients (zero where d >= dHat) and the schur complement.
__device__ __forceinline__ void pair_project_recorded(int kind, const int vv[4], const V3 x[4],
                                                      const float* __restrict__ fixed,
                                                      const float* __restrict__ m_inv, float dHat, float compliance,
                                                      long long* dx, int* nc, int* bad, PairSolve& r) {
    float mi[4], w[4];
    pair_weights(kind, vv, fixed, m_inv, mi, w);
    for (int k = 0; k < 4; ++k) r.g[k] = V3{0.0f, 0.0f, 0.0f};
    pair_solve<true>(kind, x, w, dHat, compliance, r);
    if (r.d < dHat) pair_apply(kind, vv, mi, w, r, dx, nc, bad);
}

#define SX_ZERO_G {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}}

// Candidate lists walked per query, in list order, as the reference does; the
// only variant that can write pair records (their slot order is list order).
// ---------------------------------------------------------------------------
// Edge-edge contacts: __ee_st / __ee_dy (collision_constraints_x.py:313-588)
// as the reference's commented-out callers would run them (XPBD.py:217-232,
// :266-281).  Only dtype 8 (both closest points interior) with
// |x01 x x23| > 1e-3 projects; the reference comments out the other cases.
// ---------------------------------------------------------------------------
// d_type_EE (distance.py:50-99); the triple-product test is signed, as there
__device__ int d_type_EE(V3 v0, V3 v1, V3 v2, V3 v3) {
    const V3 u = sub(v1, v0), v = sub(v3, v2), w = sub(v0, v2);
    const float a = dot(u, u), b = dot(u, v), c = dot(v, v), d = dot(u, w), e = dot(v, w);
    const float D = a * c - b * b;
    float tD = D, tN = 0.0f;
    int dc = 8;
    const float sN = b * e - c * d;
    if (sN <= 0.0f) {
        tN = e;
        tD = c;
        dc = 2;
    } else if (sN >= D) {
        tN = e + b;
        tD = c;
        dc = 5;
    } else {
        tN = a * e - b * d;
        const V3 uv = cross(u, v);
        if (tN > 0.0f && tN < tD && (dot(uv, w) < 1e-4f || dot(uv, uv) < 1.0e-20f * a * c)) {
            if (sN < D / 2.0f) {
                tN = e;
                tD = c;
                dc = 2;
            } else {
                tN = e + b;
                tD = c;
                dc = 5;
            }
        }
    }
    if (tN <= 0.0f) {
        if (-d <= 0.0f) dc = 0;
        else if (-d >= a) dc = 3;
        else dc = 6;
    } else if (tN >= tD) {
        if (-d + b <= 0.0f) dc = 1;
        else if (-d + b >= a) dc = 4;
        else dc = 7;
    }
    return dc;
}
// d_EE (distance.py:119-124): squared distance between the two lines
__device__ __forceinline__ float d_EE(V3 x0, V3 x1, V3 x2, V3 x3) {
    const V3 b = cross(sub(x1, x0), sub(x3, x2));
    const float aTb = dot(sub(x2, x0), b);
    return aTb * aTb / dot(b, b);
}
// Closed-form gradient of d_EE: u = x1-x0, v = x3-x2, r = x2-x0, n = u x v,
// s = r.n, N = n.n, d = s^2/N;
//   g0 = (-2s (n + v x r) + 2d v x n)/N,  g1 = (2s v x r - 2d v x n)/N,
//   g2 = (2s (n - r x u) + 2d n x u)/N,   g3 = (2s r x u - 2d n x u)/N.
__device__ __forceinline__ void g_EE(V3 x0, V3 x1, V3 x2, V3 x3, V3 g[4]) {
    const V3 u = sub(x1, x0), v = sub(x3, x2), r = sub(x2, x0);
    const V3 n = cross(u, v);
    const float s = dot(r, n);
    const float N = dot(n, n);
    const float iN = 1.0f / N;
    const float d = (s * s) * iN;
    const float ts = 2.0f * s, td = 2.0f * d;
    const V3 vr = cross(v, r), ru = cross(r, u), vn = cross(v, n), nu = cross(n, u);
    g[0] = scale(iN, add(scale(-ts, add(n, vr)), scale(td, vn)));
    g[1] = scale(iN, sub(scale(ts, vr), scale(td, vn)));
    g[2] = scale(iN, add(scale(ts, sub(n, ru)), scale(td, nu)));
    g[3] = scale(iN, sub(scale(ts, ru), scale(td, nu)));
}
// dtype; for dtype 8 with |x01 x x23| > 1e-3 the squared distance and, below
// dHat, its gradient; d = dHat otherwise
__device__ __forceinline__ float ee_pair(V3 x0, V3 x1, V3 x2, V3 x3, float dHat, int* dtype, V3 g[4]) {
    const int dt = d_type_EE(x0, x1, x2, x3);
    *dtype = dt;
    float d = dHat;
    if (dt == 8) {
        const V3 c = cross(sub(x0, x1), sub(x2, x3));
        if (sqrtf(dot(c, c)) > 1e-3f) {
            d = d_EE(x0, x1, x2, x3);
            if (d < dHat) g_EE(x0, x1, x2, x3, g);
        }
    }
    return d;
}

__global__ void edge_edge_classify_kernel(int n, const float* __restrict__ p12, float dHat, int* dtype, float* d,
                                          float* g12) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* p = p12 + 12 * (size_t)i;
    V3 g[4] = SX_ZERO_G;
    int dt;
    d[i] = ee_pair(V3{p[0], p[1], p[2]}, V3{p[3], p[4], p[5]}, V3{p[6], p[7], p[8]}, V3{p[9], p[10], p[11]}, dHat,
                   &dt, g);
    dtype[i] = dt;
    for (int k = 0; k < 4; ++k) {
        g12[12 * (size_t)i + 3 * k] = g[k].x;
        g12[12 * (size_t)i + 3 * k + 1] = g[k].y;
        g12[12 * (size_t)i + 3 * k + 2] = g[k].z;
    }
}

// Thread per query edge: ee_st block [0, Ed) against the static mesh's edges,
// ee_dy block [Ed, 2 Ed) against the cloth's own; for each candidate face, its
// three edges in order (vertex-sharing pairs skipped for ee_dy, XPBD.py:130-136).
__global__ void __launch_bounds__(128) edge_edge_kernel(
    int Ed, const int* __restrict__ edges_dy, const int* __restrict__ edges_st, const int* __restrict__ fe_dy,
    const int* __restrict__ fe_st, const float4* __restrict__ y4, const float4* __restrict__ xs4,
    const float* __restrict__ fixed, const float* __restrict__ m_inv, float dHat, float compliance, int cap,
    const int* __restrict__ st_c, const int* __restrict__ st_n, const int* __restrict__ dy_c,
    const int* __restrict__ dy_n, long long* dx, int* nc, PairOut po, int* status, const int* conv, int iter) {
    pdl_entry();
    if (iteration_skipped(conv, iter)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * Ed) return;
    const bool st = i < Ed;
    const int e = st ? i : i - Ed;
    int bad = 0, cnt = 0;
    if (!st || st_c != nullptr) {
        const int v0 = edges_dy[2 * e], v1 = edges_dy[2 * e + 1];
        const V3 x0 = mk(y4[v0]), x1 = mk(y4[v1]);
        const float w0 = fixed[v0] * m_inv[v0], w1 = fixed[v1] * m_inv[v1];
        const int n = min(st ? st_n[e] : dy_n[e], cap);
        for (int j = 0; j < n; ++j) {
            const int f = st ? st_c[(size_t)e * cap + j] : dy_c[(size_t)e * cap + j];
            for (int k = 0; k < 3; ++k) {
                const int e2 = st ? fe_st[3 * f + k] : fe_dy[3 * f + k];
                const int v2 = st ? edges_st[2 * e2] : edges_dy[2 * e2];
                const int v3 = st ? edges_st[2 * e2 + 1] : edges_dy[2 * e2 + 1];
                if (!st && (v0 == v2 || v0 == v3 || v1 == v2 || v1 == v3)) continue;
                const V3 x2 = mk((st ? xs4 : y4)[v2]), x3 = mk((st ? xs4 : y4)[v3]);
                V3 g[4] = SX_ZERO_G;
                int dt;
                const float d = ee_pair(x0, x1, x2, x3, dHat, &dt, g);
                if (d < dHat) {
                    float schur;
                    if (st) {
                        schur = w0 * dot(g[0], g[0]) + w1 * dot(g[1], g[1]);
                    } else {
                        const float w2 = fixed[v2] * m_inv[v2], w3 = fixed[v3] * m_inv[v3];
                        schur = ((w0 * dot(g[0], g[0]) + w1 * dot(g[1], g[1])) + w2 * dot(g[2], g[2])) +
                                w3 * dot(g[3], g[3]);
                    }
                    const float ld = (compliance * (dHat - d)) / (compliance * schur + 1.0f);
                    acc_add(dx, nc, v0, w0 * ld, g[0], &bad);
                    acc_add(dx, nc, v1, w1 * ld, g[1], &bad);
                    if (!st) {
                        acc_add(dx, nc, v2, (fixed[v2] * m_inv[v2]) * ld, g[2], &bad);
                        acc_add(dx, nc, v3, (fixed[v3] * m_inv[v3]) * ld, g[3], &bad);
                    }
                    po.rec((size_t)i, cnt, e2, dt, g, schur);
                }
            }
        }
    }
    if (po.num) po.num[i] = cnt;
    if (bad) atomicOr(status, SX_STATUS_FIXED_RANGE);
}

__global__ void __launch_bounds__(128) collision_project_kernel(
    int Vd, int Vs, const int* __restrict__ faces_dy, const int* __restrict__ faces_st,
    const float4* __restrict__ y4, const float4* __restrict__ xs4, const float* __restrict__ fixed,
    const float* __restrict__ m_inv, float dHat, float compliance, int cap, const int* __restrict__ vt_st_c,
    const int* __restrict__ vt_st_n, const int* __restrict__ vt_dy_c, const int* __restrict__ vt_dy_n,
    const int* __restrict__ tv_st_c, const int* __restrict__ tv_st_n, long long* dx, int* nc, PairOut po,
    int* status) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * Vd + Vs) return;
    int bad = 0;
    int cnt = 0;
    if (i < Vd) {
        const int vid = i;
        const int n = min(vt_st_n[vid], cap);
        const V3 x0 = mk(y4[vid]);
        for (int j = 0; j < n; ++j) {
            const int fs = vt_st_c[(size_t)vid * cap + j];
            const V3 x1 = mk(xs4[faces_st[3 * fs]]), x2 = mk(xs4[faces_st[3 * fs + 1]]),
                     x3 = mk(xs4[faces_st[3 * fs + 2]]);
            const int vv[4] = {vid, -1, -1, -1};
            const V3 x[4] = {x0, x1, x2, x3};
            PairSolve r;
            pair_project_recorded(VT_ST, vv, x, fixed, m_inv, dHat, compliance, dx, nc, &bad, r);
            if (r.d < dHat) po.rec((size_t)vid, cnt, fs, r.dt, r.g, r.schur);
        }
        if (po.num) po.num[vid] = cnt;
    } else if (i < 2 * Vd) {
        const int vid = i - Vd;
        const int n = min(vt_dy_n[vid], cap);
        for (int j = 0; j < n; ++j) {
            const int fd = vt_dy_c[(size_t)vid * cap + j];
            const int a = faces_dy[3 * fd], b = faces_dy[3 * fd + 1], c = faces_dy[3 * fd + 2];
            if (a == vid || b == vid || c == vid) continue;  // Solver.is_in_face, XPBD.py:121-127
            const int vv[4] = {vid, a, b, c};
            const V3 x[4] = {mk(y4[vid]), mk(y4[a]), mk(y4[b]), mk(y4[c])};
            PairSolve r;
            pair_project_recorded(VT_DY, vv, x, fixed, m_inv, dHat, compliance, dx, nc, &bad, r);
            po.rec((size_t)Vd + vid, cnt, fd, r.dt, r.g, r.schur);
        }
        if (po.num) po.num[Vd + vid] = cnt;
    } else {
        const int vis = i - 2 * Vd;
        const int n = min(tv_st_n[vis], cap);
        for (int j = 0; j < n; ++j) {
            const int fd = tv_st_c[(size_t)vis * cap + j];
            const int vv[4] = {-1, faces_dy[3 * fd], faces_dy[3 * fd + 1], faces_dy[3 * fd + 2]};
            const V3 x[4] = {mk(xs4[vis]), mk(y4[vv[1]]), mk(y4[vv[2]]), mk(y4[vv[3]])};
            PairSolve r;
            pair_project_recorded(TV_ST, vv, x, fixed, m_inv, dHat, compliance, dx, nc, &bad, r);
            po.rec((size_t)2 * Vd + vis, cnt, fd, r.dt, r.g, r.schur);
        }
        if (po.num) po.num[2 * Vd + vis] = cnt;
    }
    if (bad) atomicOr(status, SX_STATUS_FIXED_RANGE);
}

// ---------------------------------------------------------------------------
// Compacted pair list.  The candidate lists do not change between the Jacobi
// iterations of a substep, so once per substep they are flattened into one
// dense array of (query vertex, triangle vertices) quads, in query order,
// without the faces __vt_dy skips (incident ones); every iteration then runs
// one thread per pair.  The per-pair arithmetic is the same code as above and
// accumulation is order independent, so the result equals the per-query walk.
// Workspace: block and query totals, then meta[7] = {end of vt_st pairs, end of vt_dy
// pairs, total pairs, heads in use, heads with a bound, blocks that wrote them, the
// heads' cull_d2 as float bits}.
// ---------------------------------------------------------------------------
// Two launches, the counts and the pairs, both chains of dependent loads (count,
// candidate, its face) that a thread a query walked 20 to 30 times: eight lanes take
// a query's candidates, up to three each at once, so that most queries are one round
// of loads.  The second launch adds up the totals of the blocks before its own (up to
// PAIRS_DIRECT blocks, four loads a thread; beyond that a scan between the two).
// Count, scan and fill of a 64 x 64 sheet on a box (66 K pairs) 23.0 -> 5.9 us, of a
// 181 x 139 one on a sphere (115 K) 14.4 -> 8.2, of a 256 x 256 one (1.2 M pairs, 19
// MB written) 36.6 -> 18.3; four lanes 8.6 / 7.9 / 15.7, sixteen 5.1 / 11.8 / 26.2.
constexpr int PB = 1024, PAIR_LANES = 8, PAIR_QUERIES = PB / PAIR_LANES, PAIR_ROUNDS = 3;
constexpr int PAIRS_DIRECT = 4096;
static_assert(PB == 32 * 32, "a warp adds up the block's 32 warp totals");

// A query of the concatenated lists: cloth vertices against obstacle faces, against
// cloth faces (own: without the incident ones), obstacle vertices against cloth faces.
struct QueryList {
    int n;           // candidates
    int vid;
    bool own;
    const int* cand;
    const int* tri;  // the faces they index
};
__device__ __forceinline__ QueryList query_list(int q, int Vd, int Vs, int cap, const int* faces_dy,
                                                const int* faces_st, const int* vt_st_c, const int* vt_st_n,
                                                const int* vt_dy_c, const int* vt_dy_n, const int* tv_st_c,
                                                const int* tv_st_n) {
    if (q < Vd) return {min(vt_st_n[q], cap), q, false, vt_st_c + (size_t)q * cap, faces_st};
    if (q < 2 * Vd) return {min(vt_dy_n[q - Vd], cap), q - Vd, true, vt_dy_c + (size_t)(q - Vd) * cap, faces_dy};
    if (q < 2 * Vd + Vs)
        return {min(tv_st_n[q - 2 * Vd], cap), q - 2 * Vd, false, tv_st_c + (size_t)(q - 2 * Vd) * cap, faces_dy};
    return {0, 0, false, nullptr, nullptr};
}
// This lane's candidates j, j + 8, ... of the query below n as triangles; keep[r]
// tells whether candidate j + 8 r makes a pair.
__device__ __forceinline__ void query_round(const QueryList& l, int n, int j, int3* t, bool* keep) {
    int f[PAIR_ROUNDS];
#pragma unroll
    for (int r = 0; r < PAIR_ROUNDS; ++r) {
        keep[r] = j + PAIR_LANES * r < n;
        f[r] = keep[r] ? l.cand[j + PAIR_LANES * r] : 0;
    }
#pragma unroll
    for (int r = 0; r < PAIR_ROUNDS; ++r) {
        t[r] = make_int3(-1, -1, -1);
        if (keep[r]) t[r] = make_int3(l.tri[3 * f[r]], l.tri[3 * f[r] + 1], l.tri[3 * f[r] + 2]);
        keep[r] = keep[r] && !(l.own && (t[r].x == l.vid || t[r].y == l.vid || t[r].z == l.vid));
    }
}

__global__ void __launch_bounds__(PB, 2) pairs_count_kernel(int Vd, int Vs, int cap, const int* __restrict__ faces_dy,
                                                         const int* __restrict__ vt_st_n,
                                                         const int* __restrict__ vt_dy_c,
                                                         const int* __restrict__ vt_dy_n,
                                                         const int* __restrict__ tv_st_n, int* __restrict__ block_tot,
                                                         int* __restrict__ query_tot) {
    pdl_entry();
    __shared__ int warp_tot[PB / 32];
    const int q = blockIdx.x * PAIR_QUERIES + threadIdx.x / PAIR_LANES;
    const int lane = threadIdx.x & 31, sub = threadIdx.x & (PAIR_LANES - 1);
    const QueryList l = query_list(q, Vd, Vs, cap, faces_dy, nullptr, nullptr, vt_st_n, vt_dy_c, vt_dy_n, nullptr,
                                   tv_st_n);
    int c = 0;
    if (l.own)
        for (int j = sub; j < l.n; j += PAIR_LANES * PAIR_ROUNDS) {
            int3 t[PAIR_ROUNDS];
            bool keep[PAIR_ROUNDS];
            query_round(l, l.n, j, t, keep);
#pragma unroll
            for (int r = 0; r < PAIR_ROUNDS; ++r) c += keep[r];
        }
    __syncwarp();
#pragma unroll
    for (int o = 1; o < PAIR_LANES; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (!l.own) c = l.n;
    if (sub == 0 && q < 2 * Vd + Vs) query_tot[q] = c;
    const int w = __reduce_add_sync(0xffffffffu, sub == 0 ? c : 0);
    if (lane == 0) warp_tot[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int tot = __reduce_add_sync(0xffffffffu, warp_tot[lane]);
        if (lane == 0) block_tot[blockIdx.x] = tot;
    }
}

__global__ void __launch_bounds__(1024) pairs_scan_kernel(int nb, int* block_tot) {
    pdl_entry();
    __shared__ int s[1024];
    const int tid = threadIdx.x;
    const int per = (nb + 1023) / 1024;
    const int beg = min(tid * per, nb), end = min(beg + per, nb);
    int sum = 0;
    for (int i = beg; i < end; ++i) sum += block_tot[i];
    s[tid] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        int v = tid >= off ? s[tid - off] : 0;
        __syncthreads();
        s[tid] += v;
        __syncthreads();
    }
    int run = tid ? s[tid - 1] : 0;
    for (int i = beg; i < end; ++i) {
        int t = block_tot[i];
        block_tot[i] = run;
        run += t;
    }
}

// direct: block_tot holds the blocks' totals, else the sums before them.
__global__ void __launch_bounds__(PB, 2) pairs_fill_kernel(int Vd, int Vs, int cap, const int* __restrict__ faces_dy,
                                                        const int* __restrict__ faces_st,
                                                        const int* __restrict__ vt_st_c,
                                                        const int* __restrict__ vt_st_n,
                                                        const int* __restrict__ vt_dy_c,
                                                        const int* __restrict__ vt_dy_n,
                                                        const int* __restrict__ tv_st_c,
                                                        const int* __restrict__ tv_st_n,
                                                        const int* __restrict__ block_tot,
                                                        const int* __restrict__ query_tot, int direct, int4* pairs,
                                                        int* meta) {
    pdl_entry();
    __shared__ int warp_off[PB / 32], warp_before[PB / 32];
    const int Q = 2 * Vd + Vs;
    const int q = blockIdx.x * PAIR_QUERIES + threadIdx.x / PAIR_LANES;
    const int lane = threadIdx.x & 31, sub = threadIdx.x & (PAIR_LANES - 1), w = threadIdx.x >> 5;
    const QueryList l = query_list(q, Vd, Vs, cap, faces_dy, faces_st, vt_st_c, vt_st_n, vt_dy_c, vt_dy_n, tv_st_c,
                                   tv_st_n);
    const int c = q < Q ? query_tot[q] : 0;
    int before = 0;
    if (direct)
        for (int k = threadIdx.x; k < (int)blockIdx.x; k += PB) before += block_tot[k];
    else if (threadIdx.x == 0)
        before = block_tot[blockIdx.x];
    before = __reduce_add_sync(0xffffffffu, before);
    // pairs of the warp's queries before this one
    int off = 0, warp = 0;
#pragma unroll
    for (int k = 0; k < 32; k += PAIR_LANES) {
        const int ck = __shfl_sync(0xffffffffu, c, k);
        if (lane >= k + PAIR_LANES) off += ck;
        warp += ck;
    }
    if (lane == 0) {
        warp_off[w] = warp;
        warp_before[w] = before;
    }
    __syncthreads();
    off += __reduce_add_sync(0xffffffffu, warp_before[lane] + (lane < w ? warp_off[lane] : 0));
    if (sub == 0) {
        if (q == Vd) meta[0] = off;
        if (q == 2 * Vd) meta[1] = off;
        if (q == Q) {
            meta[2] = off;
            meta[3] = 0;  // no heads of this list yet, none of them useful
            meta[4] = 0;
            meta[5] = 0;
        }
    }
    const int most = __reduce_max_sync(0xffffffffu, l.n);
    for (int j = sub; j - sub < most; j += PAIR_LANES * PAIR_ROUNDS) {
        int3 t[PAIR_ROUNDS];
        bool keep[PAIR_ROUNDS];
        query_round(l, l.n, j, t, keep);
#pragma unroll
        for (int r = 0; r < PAIR_ROUNDS; ++r) {
            const unsigned m = __ballot_sync(0xffffffffu, keep[r]) >> (lane & ~(PAIR_LANES - 1)) &
                               ((1u << PAIR_LANES) - 1u);
            if (keep[r]) pairs[off + __popc(m & ((1u << sub) - 1u))] = make_int4(l.vid, t[r].x, t[r].y, t[r].z);
            off += __popc(m);
        }
    }
}

// Squared distance from p to the axis-aligned box of triangle (t0, t1, t2).
// The point-triangle distance of every region d_type_PT can return is at
// least this (its feature lies in the triangle), so a pair whose box distance
// exceeds dHat by a margin cannot be in contact; the pair-list sweep culls
// such pairs before the region classification when asked to.
__device__ __forceinline__ float box_d2(V3 p, V3 t0, V3 t1, V3 t2) {
    const float ex = fmaxf(fmaxf(fminf(fminf(t0.x, t1.x), t2.x) - p.x, p.x - fmaxf(fmaxf(t0.x, t1.x), t2.x)), 0.0f);
    const float ey = fmaxf(fmaxf(fminf(fminf(t0.y, t1.y), t2.y) - p.y, p.y - fmaxf(fmaxf(t0.y, t1.y), t2.y)), 0.0f);
    const float ez = fmaxf(fmaxf(fminf(fminf(t0.z, t1.z), t2.z) - p.z, p.z - fmaxf(fmaxf(t0.z, t1.z), t2.z)), 0.0f);
    return (ex * ex + ey * ey) + ez * ez;
}

// Both cull stages below rely on d_type_PT picking the region of the nearest
// feature.  It solves one 2x2 system per edge whose float32 determinant is
// about |e|^4 |n|^2 (n the face normal); for tiny or degenerate triangles that
// leaves the normal range and the classification turns arbitrary (a far point
// can get the plane region and a spurious contact, which the reference then
// applies).  The culls therefore skip only pairs of triangles whose
// determinants stay far inside the range: |n|^2 min|e|^4 > 1e-30 and
// |n|^2 max|e|^4 < 1e30.  NaN positions fail the test as well.
// The thresholds sit eight orders of magnitude inside the range, so the test
// is evaluated with fused multiply-adds: it decides only whether a pair may be
// skipped, and on classifiable triangles both decisions give the same sums.
__device__ __forceinline__ float fdot(V3 a, V3 b) { return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, a.z * b.z)); }

__device__ __forceinline__ bool classifiable(V3 a, V3 b, V3 c) {
    const V3 e0 = sub(b, a), e1 = sub(c, b), e2 = sub(a, c);
    const V3 n = {__fmaf_rn(e0.y, -e2.z, e0.z * e2.y), __fmaf_rn(e0.z, -e2.x, e0.x * e2.z),
                  __fmaf_rn(e0.x, -e2.y, e0.y * e2.x)};  // e0 x (c - a)
    const float nn = fdot(n, n);
    const float l0 = fdot(e0, e0), l1 = fdot(e1, e1), l2 = fdot(e2, e2);
    const float lo = fminf(fminf(l0, l1), l2), hi = fmaxf(fmaxf(l0, l1), l2);
    return (nn * lo) * lo > 1e-30f && (nn * hi) * hi < 1e30f;
}

// First stage: the point's squared distance to the triangle's box exceeds
// cull_d2 (a margin above dHat) on a classifiable triangle.
__device__ __forceinline__ bool box_far(V3 p, V3 a, V3 b, V3 c, float cull_d2) {
    return box_d2(p, a, b, c) > cull_d2 && classifiable(a, b, c);
}

// Separating-axis cull, the second stage after box_d2.  For any axis m the
// projection onto m/|m| is 1-Lipschitz, so dist(p, T) >= gap / |m| where gap
// is the distance from p's projection to the interval of T's vertices.  The
// axes are the face normal n = (b-a) x (c-a) and the in-plane edge normals
// e x n: together they give the distance to the edge line for a point beside
// an edge, which is what separates a flat cloth's vertex from the nearby
// triangles of its own sheet (their boxes contain it, so box_d2 is 0).  Every
// region's distance d_type_PT picks is at least dist(p, T) (a vertex, the
// edge segment its projection falls on, or the plane over the triangle), so a
// pair whose bound exceeds cull_d2 (a margin above dHat) adds nothing.  The
// bound is made safe against rounding: each projection s_k = (v_k - p) . m
// errs by less than 2.4e-7 |v_k - p|_1 |m|_1 (three products and two sums,
// plus the rounding of v_k - p), the test subtracts 1e-6 max_k |v_k - p|_1
// |m|_1 from the gap and asks for a further 1e-5 relative margin; axes with
// |m|^2 <= 1e-30 (degenerate triangles) are not used.
__device__ __forceinline__ float l1n(V3 a) { return (fabsf(a.x) + fabsf(a.y)) + fabsf(a.z); }

__device__ __forceinline__ bool far_along(V3 m, V3 da, V3 db, V3 dc, float l1, float cull_d2) {
    const float mm = dot(m, m);
    const float sa = dot(da, m), sb = dot(db, m), sc = dot(dc, m);
    const float gap = fmaxf(fminf(fminf(sa, sb), sc), -fmaxf(fmaxf(sa, sb), sc)) - 1e-6f * (l1 * l1n(m));
    return mm > 1e-30f && gap > 0.0f && gap * gap > (cull_d2 * mm) * 1.00001f;
}

__device__ __forceinline__ bool sat_far(V3 p, V3 a, V3 b, V3 c, float cull_d2) {
    const V3 da = sub(a, p), db = sub(b, p), dc = sub(c, p);
    const float l1 = fmaxf(fmaxf(l1n(da), l1n(db)), l1n(dc));
    const V3 eab = sub(db, da), ebc = sub(dc, db), eca = sub(da, dc);
    const V3 n = cross(eab, sub(dc, da));
    return classifiable(a, b, c) &&
           (far_along(n, da, db, dc, l1, cull_d2) || far_along(cross(eab, n), da, db, dc, l1, cull_d2) ||
            far_along(cross(ebc, n), da, db, dc, l1, cull_d2) || far_along(cross(eca, n), da, db, dc, l1, cull_d2));
}

// One pair of the list: positions of its four vertices and the projection of
// its kind (vt_st, vt_dy or tv_st by list position).
struct PairCtx {
    const int4* __restrict__ pairs;
    const float4* __restrict__ y4;
    const float4* __restrict__ xs4;
    const float* __restrict__ fixed;
    const float* __restrict__ m_inv;
    float dHat, compliance;
    long long* dx;
    int* nc;
    int st_end, dy_end;
};

__device__ __forceinline__ void pair_points(const PairCtx& c, int t, int4 pr, V3 x[4]) {
    const bool st = t < c.st_end, tv = t >= c.dy_end;
    x[0] = mk((tv ? c.xs4 : c.y4)[pr.x]);
    const float4* tri = st ? c.xs4 : c.y4;
    x[1] = mk(tri[pr.y]);
    x[2] = mk(tri[pr.z]);
    x[3] = mk(tri[pr.w]);
}

// ---------------------------------------------------------------------------
// Skipping the vertex-vs-cloth pairs that cannot have come into reach.
//
// Nearly all of those pairs are a vertex and a triangle of its own sheet a few
// edges away: never in contact, and in every iteration tested again, which is
// what a contact sweep over a large sheet costs.  Vertices move little within a
// substep, so once per substep (sx_contact_pairs_heads, after the first
// iteration) each chunk of 32 consecutive pairs gets a head: a motion mu below
// which none of its pairs can come into reach, and the blocks of 32 vertices its
// pairs touch.  The sweeps keep, per block, the largest squared displacement since
// then (SweepTrack), and a projection given the heads passes over every chunk all
// of whose blocks moved at most mu.  The chunk's other pairs are tested as ever.
//
// mu of a pair: with a lower bound D on its distance (the box's, and the gap
// along the separating axes of sat_far, rounding subtracted as there) and c =
// sqrt(cull_d2), motions of at most mu = (D - c) / 2 of its four vertices keep
// the point farther than c from the triangle.  That a region's distance is at
// least the true one needs a classifiable triangle (see classifiable), so mu is
// also at most an eighth of the triangle's least altitude h, and the triangle has
// to satisfy |n|^2 min|e|^4 > 1e-26 and |n|^2 max|e|^4 < 1e26: edges then change
// by at most h / 4 <= a quarter of themselves and |n| by at most 9/16 of itself,
// so the two products stay within factors 0.06 and 6 of what they were, inside
// classifiable's 1e-30 and 1e30.  A skipped pair is therefore one that adds
// nothing, and the sums are the same bit for bit.
//
// Head: 16 words, {mu^2 or -1, up to 15 blocks (the first repeated)}; -1 when a
// pair has no such mu or the chunk touches more blocks (a mesh whose numbering
// has no locality: its chunks are tested as before).
// ---------------------------------------------------------------------------
constexpr int HEAD_WORDS = 16;

__device__ __forceinline__ float axis_gap(V3 m, V3 da, V3 db, V3 dc, float l1) {
    const float mm = dot(m, m);
    const float sa = dot(da, m), sb = dot(db, m), sc = dot(dc, m);
    const float gap = fmaxf(fminf(fminf(sa, sb), sc), -fmaxf(fmaxf(sa, sb), sc)) - 1e-6f * (l1 * l1n(m));
    return mm > 1e-30f ? gap * rsqrtf(mm) : 0.0f;
}
// -1: none
__device__ __forceinline__ float pair_reach_motion(V3 p, V3 a, V3 b, V3 c, float cull) {
    const V3 da = sub(a, p), db = sub(b, p), dc = sub(c, p);
    const float l1 = fmaxf(fmaxf(l1n(da), l1n(db)), l1n(dc));
    const V3 eab = sub(db, da), ebc = sub(dc, db), eca = sub(da, dc);
    const V3 n = cross(eab, sub(dc, da));
    const float nn = dot(n, n);
    const float l0 = dot(eab, eab), l2 = dot(ebc, ebc), l3 = dot(eca, eca);
    const float lo = fminf(fminf(l0, l2), l3), hi = fmaxf(fmaxf(l0, l2), l3);
    float d = sqrtf(box_d2(p, a, b, c));
    d = fmaxf(d, axis_gap(n, da, db, dc, l1));
    d = fmaxf(d, axis_gap(cross(eab, n), da, db, dc, l1));
    d = fmaxf(d, axis_gap(cross(ebc, n), da, db, dc, l1));
    d = fmaxf(d, axis_gap(cross(eca, n), da, db, dc, l1));
    // (a NaN in p is its block's motion in every tracked sweep)
    const float mu = fminf(0.499f * (d * 0.9999f - cull * 1.0001f), 0.12f * sqrtf(nn / hi));
    return mu > 0.0f && (nn * lo) * lo > 1e-26f && (nn * hi) * hi < 1e26f ? mu : -1.0f;
}

// meta[4] counts the heads with a mu, meta[5] the blocks that have added theirs;
// the last one puts the heads to use, meta[3] = 1, when more than half have one.
// With fewer than min_pairs vertex-vs-cloth pairs the projection costs less than
// this, and the heads stay unwritten.
__global__ void __launch_bounds__(256) pairs_heads_kernel(int V, int* meta, const int4* __restrict__ pairs,
                                                          const float4* __restrict__ y4, float cull_d2, int min_pairs,
                                                          float4* __restrict__ ref, unsigned* __restrict__ moved,
                                                          int* __restrict__ heads) {
    pdl_entry();
    const int first = meta[0], last = meta[1];
    const bool on = last - first >= min_pairs && cull_d2 > 0.0f;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    if (!on) {
        if (tid == 0) meta[3] = 0;
        return;
    }
    if (tid == 0) meta[6] = __float_as_int(cull_d2);
    for (int v = tid; v < V; v += nt) {
        ref[v] = y4[v];
        if ((v & 31) == 0) moved[v >> 5] = 0u;
    }
    const int lane = threadIdx.x & 31;
    const float cull = sqrtf(cull_d2);
    const int nchunks = (last - first + 31) / 32;
    int useful = 0;
    for (int c = tid >> 5; c < nchunks; c += nt >> 5) {
        const int t = first + 32 * c + lane;
        const bool valid = t < last;
        int b[4] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff};
        float mu = INFINITY;
        if (valid) {
            const int4 pr = pairs[t];
            mu = pair_reach_motion(mk(y4[pr.x]), mk(y4[pr.y]), mk(y4[pr.z]), mk(y4[pr.w]), cull);
            b[0] = pr.x >> 5;
            b[1] = pr.y >> 5;
            b[2] = pr.z >> 5;
            b[3] = pr.w >> 5;
        }
        int word = 0;
        if (__all_sync(0xffffffffu, mu > 0.0f)) {
            const float least = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(mu)));
            // the distinct blocks in ascending order, block k to lane k + 1
            int prev = -1, n = 0;
            for (;; ++n) {
                int next = 0x7fffffff;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (b[k] > prev) next = min(next, b[k]);
                next = __reduce_min_sync(0xffffffffu, next);
                if (next == 0x7fffffff || n == HEAD_WORDS - 1) {
                    if (next != 0x7fffffff) n = HEAD_WORDS;  // too many
                    break;
                }
                if (lane == n + 1) word = next;
                prev = next;
            }
            const int one = __shfl_sync(0xffffffffu, word, 1);
            if (lane > n) word = one;
            if (lane == 0) {
                word = __float_as_int(n == HEAD_WORDS ? -1.0f : (least * least) * 0.999f);
                if (n != HEAD_WORDS) ++useful;
            }
        } else if (lane == 0) {
            word = __float_as_int(-1.0f);
        }
        if (lane < HEAD_WORDS) heads[(size_t)c * HEAD_WORDS + lane] = word;
    }
    if (useful) atomicAdd(meta + 4, useful);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(meta + 5, 1) == (int)gridDim.x - 1)
        meta[3] = 2 * atomicAdd(meta + 4, 0) > nchunks ? 1 : 0;
}
// whether a chunk has to be tested
__device__ __forceinline__ bool head_moved(const int* __restrict__ heads, const unsigned* __restrict__ moved, int c) {
    const int4* h = reinterpret_cast<const int4*>(heads + (size_t)c * HEAD_WORDS);
    const int4 q0 = h[0], q1 = h[1], q2 = h[2], q3 = h[3];
    const float mu2 = __int_as_float(q0.x);
    if (!(mu2 > 0.0f)) return true;
    const int id[15] = {q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z, q3.w};
    unsigned m = 0u;
#pragma unroll
    for (int k = 0; k < 15; ++k) m = max(m, moved[id[k]]);
    return !(__uint_as_float(m) <= mu2);
}

constexpr int PP_BLOCK = 256;

// With the cull on, most pairs end at the box test, most of the rest at the
// separating-axis test, and the few that remain would leave a warp mostly idle
// through the region classification.  Each warp therefore box-tests U x 32
// pairs at a time (all their records first, then all their vertex gathers, so
// U batches of loads are in flight) and appends the survivors to a stack in
// shared memory (ballot); 32 at a time they go through the separating-axis
// test onto a second stack, and 32 at a time from there through the
// projection, every stage with all lanes busy.  The projection stands in one
// place of the loop, which keeps the kernel's code and registers small.  The
// contact sums are order independent, so U and the stacking change the speed
// only.
//
// PIPE: the two kinds against the obstacle (vertex vs obstacle face, obstacle
// vertex vs cloth face) are few pairs of which most reach the classification;
// the last warps take them one per lane from the box test straight to the
// projection, on the positions already in registers.  The vertex-vs-cloth pairs then go through the stages
// above, with the next step's pair records loaded while the current step's
// positions are gathered, so that a warp waits on one round trip per step
// instead of two.
//
// HEADED: a warp first looks at the heads of its chunks, 32 of them together
// (chunks gw, gw + nw, ...: neighbours, which move together, lie on different
// warps), and takes only those that moved, or all of them where the heads are not
// in use (a body with both loops spills and costs such a list 0.3 us).
template <int U, bool PIPE, bool HEADED>
__device__ __forceinline__ void pairs_project_body(const PairCtx& c, int P, bool in_use, float cull_d2, int* s1,
                                                   int* s2, int* status, const int* __restrict__ heads,
                                                   const unsigned* __restrict__ moved) {
    const int4* __restrict__ pairs = c.pairs;
    const float4* __restrict__ y4 = c.y4;
    const int st_end = c.st_end, dy_end = c.dy_end;
    const bool cull = cull_d2 > 0.0f;  // without it every pair is classified
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    int n1 = 0, n2 = 0;  // warp-uniform
    int bad = 0;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const bool split = HEADED || (PIPE && cull);
    const int first = split ? st_end : 0, last = split ? dy_end : P, chunk = cull ? 32 * U : 32;
    // the obstacle kinds go to the last warps, which have the fewest chunks
    const int H = split ? st_end + (P - dy_end) : 0;
    int h0 = (nw - 1 - gw) * 32, base = HEADED ? last : first + gw * chunk;
    auto push = [&](int* s, int& n, int t, bool keep) {
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) s[n + __popc(m & below)] = t;
        n += __popc(m);
    };
    const int nchunks = HEADED ? (dy_end - st_end + 31) / 32 : 0;
    int c0 = gw;  // the first chunk of the next look
    unsigned todo = 0u;
    int4 nx[U];
    if (split && !HEADED) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = base + 32 * u + lane;
            nx[u] = t < last ? pairs[t] : make_int4(0, 0, 0, 0);
        }
    }
    for (;;) {
        int t = -1;  // the pair this lane projects
        int4 pr = make_int4(0, 0, 0, 0);
        V3 x[4];
        if (h0 < H) {
            const int h = h0 + lane;
            if (h < H) {
                t = h < st_end ? h : dy_end + (h - st_end);
                pr = pairs[t];
                pair_points(c, t, pr, x);
                if (box_far(x[0], x[1], x[2], x[3], cull_d2)) t = -1;
            }
            h0 += nw * 32;
        } else {
            // fill the second stack to at least 32 entries, or to what is left
            bool more = true;
            while (n2 < 32 && more) {
                if (n1 >= 32 || (n1 > 0 && base >= last && (!HEADED || (todo == 0u && c0 >= nchunks)))) {
                    // the top of s1 through the separating-axis test onto s2
                    const int cnt = n1 < 32 ? n1 : 32;
                    const int q = lane < cnt ? s1[n1 - cnt + lane] : -1;
                    bool keep = false;
                    if (q >= 0) {
                        V3 z[4];
                        pair_points(c, q, pairs[q], z);
                        keep = !sat_far(z[0], z[1], z[2], z[3], cull_d2);
                    }
                    n1 -= cnt;
                    push(s2, n2, q, keep);
                } else if (HEADED && c0 < nchunks && todo == 0u) {
                    const int ch = c0 + lane * nw;
                    todo = __ballot_sync(0xffffffffu, ch < nchunks && (!in_use || head_moved(heads, moved, ch)));
                    c0 += 32 * nw;
                } else if (!cull && base < last) {
                    push(s2, n2, base + lane, base + lane < last);
                    base += nw * chunk;
                } else if ((HEADED && todo != 0u) || base < last) {
                    // the next U x 32 pairs (with heads: U moved chunks)
                    int q[U];
                    V3 z[U][4];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        q[u] = base + 32 * u + lane;
                        if (HEADED) {
                            q[u] = dy_end;
                            if (todo != 0u) q[u] = st_end + 32 * (c0 + (__ffs(todo) - 33) * nw) + lane;
                            todo &= todo - 1u;
                            nx[u] = q[u] < dy_end ? pairs[q[u]] : make_int4(0, 0, 0, 0);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (PIPE) {
                            z[u][0] = mk(y4[nx[u].x]);
                            z[u][1] = mk(y4[nx[u].y]);
                            z[u][2] = mk(y4[nx[u].z]);
                            z[u][3] = mk(y4[nx[u].w]);
                        } else if (q[u] < last) {
                            pair_points(c, q[u], pairs[q[u]], z[u]);
                        }
                    }
                    if (PIPE && !HEADED) {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int t = base + nw * chunk + 32 * u + lane;
                            nx[u] = t < last ? pairs[t] : make_int4(0, 0, 0, 0);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        push(s1, n1, q[u], q[u] < last && !box_far(z[u][0], z[u][1], z[u][2], z[u][3], cull_d2));
                    if (!HEADED) base += nw * chunk;
                } else {
                    more = false;
                }
                __syncwarp();
            }
            if (n2 == 0) break;
            const int cnt = n2 < 32 ? n2 : 32;
            if (lane < cnt) {
                t = s2[n2 - cnt + lane];
                pr = pairs[t];
                pair_points(c, t, pr, x);
            }
            n2 -= cnt;
            __syncwarp();
        }
        if (t >= 0)
            pair_project(t < st_end ? VT_ST : t < dy_end ? VT_DY : TV_ST, pr, x, c.fixed, c.m_inv, c.dHat,
                         c.compliance, c.dx, c.nc, &bad);
    }
    if (bad) atomicOr(status, SX_STATUS_FIXED_RANGE);
}

template <int U, int MINB, bool PIPE, bool HEADED>
__global__ void __launch_bounds__(PP_BLOCK, MINB) pairs_project_kernel(const int* __restrict__ meta,
                                                                       const int4* __restrict__ pairs,
                                                                       const float4* __restrict__ y4,
                                                                       const float4* __restrict__ xs4,
                                                                       const float* __restrict__ fixed,
                                                                       const float* __restrict__ m_inv, float dHat,
                                                                       float compliance, float cull_d2, long long* dx,
                                                                       int* nc, int* status, const int* conv,
                                                                       int iter, const int* __restrict__ heads,
                                                                       const unsigned* __restrict__ moved) {
    pdl_entry();
    if (iteration_skipped(conv, iter)) return;
    const PairCtx c{pairs, y4, xs4, fixed, m_inv, dHat, compliance, dx, nc, meta[0], meta[1]};
    __shared__ int box_stack[PP_BLOCK / 32][32 * U + 32];
    __shared__ int sat_stack[PP_BLOCK / 32][64];
    int* s1 = box_stack[threadIdx.x >> 5];
    int* s2 = sat_stack[threadIdx.x >> 5];
    // heads bound the motion that brings a pair within their own cull distance
    const bool in_use = HEADED && heads_in_use(meta) != 0 && cull_d2 <= __int_as_float(meta[6]);
    pairs_project_body<U, PIPE, HEADED>(c, meta[2], in_use, cull_d2, s1, s2, status, heads, moved);
}

// update_dx (XPBD.py:384-387) from the fixed-point accumulators; clears them.
// One vertex a thread: four a thread (their counts in one load, or strided by
// 32) saves waves but serialises the corrections of a resting cloth's
// neighbouring vertices; a frame of 96 cloths took 9.45 instead of 8.44 ms.
__global__ void collision_apply_kernel(int V, float4* __restrict__ y4, const float* __restrict__ fixed,
                                       long long* __restrict__ dx, int* __restrict__ nc, const int* conv, int iter) {
    pdl_entry();
    if (iteration_skipped(conv, iter)) return;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const int c = nc[v];
        if (c > 0) {
            const float cf = (float)c;
            const float f = fixed[v];
            float4 y = y4[v];
            y.x = y.x + f * (from_fix(dx[3 * v]) / cf);
            y.y = y.y + f * (from_fix(dx[3 * v + 1]) / cf);
            y.z = y.z + f * (from_fix(dx[3 * v + 2]) / cf);
            y4[v] = y;
            dx[3 * v] = 0;
            dx[3 * v + 1] = 0;
            dx[3 * v + 2] = 0;
            nc[v] = 0;
        }
    }
}

// one resident wave at most (the kernels above walk their range)
template <typename K>
inline int capped_grid(K kernel, long long n, int block) {
    const int g = grid_for(n, block), cap = resident_blocks(kernel, block);
    return g < cap ? g : cap;
}

static void launch_apply(int V, float4* y4, const float* fixed, long long* dx, int* nc, const int* conv, int iter,
                         cudaStream_t s) {
    launch(collision_apply_kernel, conv ? capped_grid(collision_apply_kernel, V, 256) : grid_for(V, 256), 256, 0, s, V,
           y4, fixed, dx, nc, conv, iter);
}

// ---------------------------------------------------------------------------
// Batched independent cloths, each with its own static obstacle.
//
// Instances are concatenated with per-instance offset tables, as the
// reference concatenates meshes (framework/meshio/concat.py:11-58), but each
// instance keeps its own pair of cell BVHs' semantics: a query only meets its
// own instance's faces, and the candidate set of a query is what
// traverse_cell_bvh_single (lbvh_cell.py:662-714) returns over that
// instance's grid -- every face whose padded box overlaps the query box,
// unless the query centre falls past the last cell of the grid
// (lbvh_cell.py:665).  With at most 32 obstacle faces per instance the
// vertex-vs-obstacle candidates of a vertex fit a 32-bit mask; obstacle
// vertices list their cloth candidates in ascending face order.  Contact sums
// are order independent, so the result equals running every instance through
// the single-cloth solver with self contact off.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned f2ord_c(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f_c(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// AABB of each segment of a point array (one block per segment), +- padding,
// with the reference's 1e5 initial bounds (meshTaichiWrapper.py:335-347).  A
// block reads a segment of some 10 000 points alone, so it is bound by the
// round trips of its loads: 1024 threads with four in flight each (24 cloths of
// up to 128 x 128: 34 us with 256 threads, one load each).
constexpr int SEG_BLOCK = 1024;
__global__ void __launch_bounds__(SEG_BLOCK) segment_aabb_kernel(const float4* __restrict__ p4,
                                                                 const int* __restrict__ seg, float pad,
                                                                 float* __restrict__ box6) {
    pdl_entry();
    const int s = blockIdx.x;
    float lo[3] = {1e5f, 1e5f, 1e5f}, hi[3] = {-1e5f, -1e5f, -1e5f};
    const int e = seg[s + 1];
    for (int i = seg[s] + threadIdx.x; i < e; i += 4 * SEG_BLOCK) {
        float4 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = i + j * SEG_BLOCK < e ? p4[i + j * SEG_BLOCK] : make_float4(NAN, NAN, NAN, 0.0f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // fminf and fmaxf pass over a NaN
            lo[0] = fminf(lo[0], p[j].x); lo[1] = fminf(lo[1], p[j].y); lo[2] = fminf(lo[2], p[j].z);
            hi[0] = fmaxf(hi[0], p[j].x); hi[1] = fmaxf(hi[1], p[j].y); hi[2] = fmaxf(hi[2], p[j].z);
        }
    }
    __shared__ unsigned red[6];
    if (threadIdx.x < 6) red[threadIdx.x] = threadIdx.x < 3 ? f2ord_c(1e5f) : f2ord_c(-1e5f);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const unsigned l = __reduce_min_sync(0xffffffffu, f2ord_c(lo[k]));
        const unsigned h = __reduce_max_sync(0xffffffffu, f2ord_c(hi[k]));
        if ((threadIdx.x & 31) == 0) {
            atomicMin(red + k, l);
            atomicMax(red + 3 + k, h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const float v = ord2f_c(red[threadIdx.x]);
        box6[6 * s + threadIdx.x] = threadIdx.x < 3 ? v - pad : v + pad;
    }
}

// The reference's skip test of a query box against a grid built on box6.
__device__ __forceinline__ bool query_skipped(V3 a, V3 b, const float* box6) {
    const V3 pos = scale(0.5f, add(a, b));
    const V3 org{box6[0], box6[1], box6[2]};
    const V3 cs{(box6[3] - box6[0]) / (float)kGridRes, (box6[4] - box6[1]) / (float)kGridRes,
                (box6[5] - box6[2]) / (float)kGridRes};
    const int ix = f2i_sat((pos.x - org.x) / cs.x), iy = f2i_sat((pos.y - org.y) / cs.y),
              iz = f2i_sat((pos.z - org.z) / cs.z);
    const int cid =
        (int)((unsigned)ix * (unsigned)(kGridRes * kGridRes) + (unsigned)iy * (unsigned)kGridRes + (unsigned)iz);
    return cid > kNumCells - 1;
}

__global__ void batched_vt_st_broad_kernel(int V, const float4* __restrict__ y4, const int* __restrict__ vinst,
                                           const float* __restrict__ ob_box6, const int* __restrict__ ob_fptr,
                                           const float4* __restrict__ ob_fmin4, const float4* __restrict__ ob_fmax4,
                                           float pad, unsigned* __restrict__ vmask) {
    pdl_entry();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int inst = vinst[v];
    const V3 p = mk(y4[v]);
    const V3 a{p.x - pad, p.y - pad, p.z - pad}, b{p.x + pad, p.y + pad, p.z + pad};
    unsigned m = 0;
    if (!query_skipped(a, b, ob_box6 + 6 * inst)) {
        const int f0 = ob_fptr[inst], f1 = ob_fptr[inst + 1];
        for (int f = f0; f < f1; ++f)
            if (overlap(a, b, mk(ob_fmin4[f]), mk(ob_fmax4[f]))) m |= 1u << (f - f0);
    }
    vmask[v] = m;
}

// one warp per obstacle vertex; candidates appended in ascending face order.
// The lanes first test the boxes of 32 chunks of 32 faces (cl_cmin4/cmax4,
// chunk c = faces 32c .. 32c+31, a superset of every face box in it), then
// test the faces of the chunks that overlap, in order.
__global__ void batched_tv_st_broad_kernel(int S, const float4* __restrict__ xs4, const int* __restrict__ svinst,
                                           const float* __restrict__ cl_box6, const int* __restrict__ cl_fptr,
                                           const float4* __restrict__ cl_fmin4, const float4* __restrict__ cl_fmax4,
                                           const float4* __restrict__ cl_cmin4, const float4* __restrict__ cl_cmax4,
                                           float pad, int cap, int* __restrict__ cand, int* __restrict__ num,
                                           int* status) {
    pdl_entry();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= S) return;
    const int inst = svinst[w];
    const V3 p = mk(xs4[w]);
    const V3 a{p.x - pad, p.y - pad, p.z - pad}, b{p.x + pad, p.y + pad, p.z + pad};
    int count = 0;
    if (!query_skipped(a, b, cl_box6 + 6 * inst)) {
        const int f0 = cl_fptr[inst], f1 = cl_fptr[inst + 1];
        const int c0 = f0 >> 5, c1 = (f1 + 31) >> 5;  // chunks touching [f0, f1)
        // four batches of chunk boxes in flight: a warp alone reads its cloth's
        constexpr int N = 4;
        for (int cb0 = c0; cb0 < c1; cb0 += 32 * N) {
            float4 lo[N], hi[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int c = cb0 + 32 * i + lane;
                lo[i] = c < c1 ? cl_cmin4[c] : make_float4(INFINITY, INFINITY, INFINITY, 0.0f);
                hi[i] = c < c1 ? cl_cmax4[c] : make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int cb = cb0 + 32 * i;
                const bool near = cb + lane < c1 && overlap(a, b, mk(lo[i]), mk(hi[i]));
                unsigned hits = __ballot_sync(0xffffffffu, near);
                while (hits) {  // warp-uniform, ascending chunks
                    const int ch = cb + __ffs(hits) - 1;
                    hits &= hits - 1u;
                    const int f = 32 * ch + lane;
                    const bool hit = f >= f0 && f < f1 && overlap(a, b, mk(cl_fmin4[f]), mk(cl_fmax4[f]));
                    const unsigned ball = __ballot_sync(0xffffffffu, hit);
                    const int slot = count + __popc(ball & ((1u << lane) - 1u));
                    if (hit && slot < cap) cand[(size_t)w * cap + slot] = f;
                    count += __popc(ball);
                }
            }
        }
    }
    if (lane == 0) {
        num[w] = count;
        if (count > cap) atomicOr(status, SX_STATUS_CAND_OVERFLOW);
    }
}

// The candidates of a substep as one dense list of quads, in no particular
// order (contact sums are order independent): (vertex, obstacle triangle) for
// the set bits of the vertices' face masks, (~obstacle vertex, cloth triangle)
// for the obstacle vertices' lists.  *count is the number found, also past the
// capacity; the list is then not used.
__global__ void __launch_bounds__(256) batched_list_kernel(int V, int S, const unsigned* __restrict__ vmask,
                                                           const int* __restrict__ vinst,
                                                           const int* __restrict__ ob_fptr,
                                                           const int* __restrict__ ob_faces,
                                                           const int* __restrict__ tv_cand,
                                                           const int* __restrict__ tv_num, int cap,
                                                           const int* __restrict__ cl_faces, int4* list,
                                                           long long capacity, unsigned long long* count) {
    pdl_entry();
    const int lane = threadIdx.x & 31;
    const long long nv = ((long long)V + 31) / 32 * 32, total = nv + (long long)S * cap;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i - lane >= total) return;
    unsigned mask = 0u;
    const int* face = nullptr;  // the first candidate's triangle
    int who = 0;
    if (i < V) {
        mask = vmask[i];
        who = (int)i;
        if (mask) face = ob_faces + 3 * (size_t)ob_fptr[vinst[i]];
    } else if (i >= nv && i < total) {
        const long long h = i - nv;
        const int s = (int)(h / cap), j = (int)(h - (long long)s * cap);
        if (j < tv_num[s]) {
            mask = 1u;
            who = ~s;
            face = cl_faces + 3 * (size_t)tv_cand[h];
        }
    }
    if (!__any_sync(0xffffffffu, mask != 0u)) return;
    const int k = __popc(mask);
    int incl = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    unsigned long long at = 0;
    if (lane == 31) at = atomicAdd(count, (unsigned long long)incl);
    at = __shfl_sync(0xffffffffu, at, 31) + (unsigned long long)(incl - k);
    for (unsigned r = mask; r != 0u; r &= r - 1u, ++at) {
        const int* f = face + 3 * (__ffs(r) - 1);
        if (at < (unsigned long long)capacity) list[at] = make_int4(who, f[0], f[1], f[2]);
    }
}

// Obstacle contacts of one iteration.  A candidate is an (obstacle vertex,
// cloth face) slot or a set bit of a cloth vertex's face mask; few vertices have
// any, and a corner of an obstacle under a lying cloth has as many as its list
// holds.  One thread per vertex would walk such a list alone (40 dependent
// classifications: 99 us per launch on 24 cloths lying on their boxes, 160 000
// vertices); here a warp tests candidates 32 at a time with the pair list's
// culls (box_far, sat_far: of a box side's two triangles most vertices reach
// one) and projects the survivors 32 at a time.  With the substep's list
// (batched_list_kernel) the candidates are dealt evenly and one load away from
// their positions; without it, or when it overflowed, the warps take 32 slots of
// the obstacle vertices' lists, then 32 cloth vertices at a time, and lay the
// set bits end to end themselves (24 cloths 19 us against 9.6 with the list, 96
// cloths 40 against 17.5 per launch, caches cold).
// Contact sums are order independent.
constexpr int BC_BLOCK = 256, BC_PER_SM = 2;

__global__ void __launch_bounds__(BC_BLOCK, BC_PER_SM) batched_contacts_kernel(
    int V, int S, const float4* __restrict__ y4, const float* __restrict__ fixed, const float* __restrict__ m_inv,
    const int* __restrict__ vinst, const int* __restrict__ ob_fptr, const int* __restrict__ ob_faces,
    const float4* __restrict__ xs4, const unsigned* __restrict__ vmask, const int* __restrict__ tv_cand,
    const int* __restrict__ tv_num, int cap, const int* __restrict__ cl_faces, float dHat, float compliance,
    const int4* __restrict__ list, long long capacity, const unsigned long long* __restrict__ count, long long* dx,
    int* nc, int* status, const int* conv, int iter) {
    pdl_entry();
    if (iteration_skipped(conv, iter)) return;
    __shared__ unsigned short items[BC_BLOCK / 32][32 * 32];  // the current task's (lane, face bit)s
    __shared__ int4 stack[BC_BLOCK / 32][64];                 // quads past the culls
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned short* it = items[threadIdx.x >> 5];
    int4* st = stack[threadIdx.x >> 5];
    const long long gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const float cull_d2 = dHat * 1.0625f;
    const unsigned long long found = list != nullptr ? *count : ~0ull;
    const bool listed = found <= (unsigned long long)capacity;
    const long long slots = listed ? (long long)found : (long long)S * cap;
    long long h0 = gw * 32;  // first list entry or slot of the warp's next task
    // vertex tasks from the other end, so that they start on the warps without list slots
    const long long ntasks = listed ? 0 : ((long long)V + 31) / 32;
    long long task = nw - 1 - gw;
    unsigned m[4] = {0u, 0u, 0u, 0u};  // masks of the tasks task, task + nw, ...
    int held = 0;                      // of them not yet laid out
    int v0 = 0, T = 0, pos = 0, n = 0, bad = 0;

    auto points = [&](int4 c, V3 x[4]) {
        const bool tv = c.x < 0;
        const float4* tri = tv ? y4 : xs4;
        x[0] = mk(tv ? xs4[~c.x] : y4[c.x]);
        x[1] = mk(tri[c.y]);
        x[2] = mk(tri[c.z]);
        x[3] = mk(tri[c.w]);
    };
    auto quad = [](int who, const int* f) { return make_int4(who, f[0], f[1], f[2]); };
    for (;;) {
        bool more = true;
        while (n < 32 && more) {
            int4 c = make_int4(0, 0, 0, 0);
            bool have = false;
            if (h0 < slots) {
                const long long h = h0 + lane;
                if (h < slots && listed) {
                    c = list[h];
                    have = true;
                } else if (h < slots) {
                    const int s = (int)(h / cap), j = (int)(h - (long long)s * cap);
                    if (j < tv_num[s]) {
                        c = quad(~s, cl_faces + 3 * (size_t)tv_cand[h]);
                        have = true;
                    }
                }
                h0 += nw * 32;
            } else if (pos < T) {
                if (pos + lane < T) {
                    const int q = it[pos + lane], v = v0 + (q >> 5);
                    c = quad(v, ob_faces + 3 * (size_t)(ob_fptr[vinst[v]] + (q & 31)));
                    have = true;
                }
                pos += 32;
            } else if (held > 0) {
                // the next task's candidates, end to end
                const unsigned mask = m[0];
                m[0] = m[1];
                m[1] = m[2];
                m[2] = m[3];
                v0 = (int)(task * 32);
                task += nw;
                --held;
                T = pos = 0;
                if (__any_sync(0xffffffffu, mask != 0u)) {
                    const int k = __popc(mask);
                    int incl = k;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    T = __shfl_sync(0xffffffffu, incl, 31);
                    int at = incl - k;
                    for (unsigned r = mask; r != 0u; r &= r - 1u) it[at++] = (unsigned short)(lane * 32 + __ffs(r) - 1);
                    __syncwarp();
                }
                continue;
            } else if (task < ntasks) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const long long v = (task + i * nw) * 32 + lane;
                    m[i] = v < V ? vmask[v] : 0u;
                    if (task + i * nw < ntasks) held = i + 1;
                }
                continue;
            } else {
                more = false;
            }
            if (have) {
                V3 x[4];
                points(c, x);
                have = !box_far(x[0], x[1], x[2], x[3], cull_d2) && !sat_far(x[0], x[1], x[2], x[3], cull_d2);
            }
            const unsigned hits = __ballot_sync(0xffffffffu, have);
            if (have) st[n + __popc(hits & below)] = c;
            n += __popc(hits);
            __syncwarp();
        }
        if (n == 0) break;
        const int cnt = n < 32 ? n : 32;
        if (lane < cnt) {
            const int4 c = st[n - cnt + lane];
            V3 x[4];
            points(c, x);
            pair_project(c.x < 0 ? TV_ST : VT_ST, c, x, fixed, m_inv, dHat, compliance, dx, nc, &bad);
        }
        n -= cnt;
        __syncwarp();
    }
    if (bad) atomicOr(status, SX_STATUS_FIXED_RANGE);
}

// ---------------------------------------------------------------------------
// Persistent batched substep.  One launch runs a whole substep of every
// instance: each CTA takes instances from a queue (largest first) and runs,
// for its instance alone, the cloth box and face boxes on x, optionally the
// prediction, all Jacobi iterations (sweep; in the first, the obstacle broad
// phase; obstacle contacts; update_dx) and the velocity update, with block
// barriers between the phases -- an instance never reads another's vertices,
// so no grid-wide synchronisation is needed.  The instance's positions and
// adjacency stay in L1/L2 across its iterations instead of streaming the
// whole batch from HBM in every sweep.  Every phase evaluates the same
// expressions as the grid-wide kernels (sweep_vertex, pair_project,
// the broad-phase tests, update_dx, compute_velocity +
// update_x), and contact sums are order independent, so the result equals the
// graph of grid-wide launches bit for bit.  Chunk boxes (32 faces) are
// aligned to each instance's first face (cptr); they only select which faces
// are tested, and the faces are tested in ascending order either way.
// The queue counter is reset by the last CTA to finish.
// ---------------------------------------------------------------------------
struct BatchedSubstepArgs {
    int n_inst, n_iter, predict, cap;
    const int *order, *vptr, *fptr, *cptr, *optr, *ob_fptr;
    float4 *x4, *ya, *yb, *v4;
    const float *fixed, *m_inv;
    const int* adj_ptr;
    const int2* adj;
    const short* nbr16;      // packed adjacency, or null
    const unsigned* rest32;
    const int *faces, *ob_faces;
    const float4* xs4;
    float4 *fmin4, *fmax4, *cmin4, *cmax4;
    float* cl_box6;
    const float* ob_box6;
    const float4 *ob_fmin4, *ob_fmax4;
    unsigned* vmask;
    int *tv_cand, *tv_num;
    long long* dx;
    int* nc;
    int *status, *queue;
    float pad, dt, gx, gy, gz, ks, kb, dHat, compliance, damping;
};

// Cluster plumbing of the persistent substep: with CL > 1 an instance is
// processed by a thread-block cluster of CL CTAs (one instance per cluster
// instead of per CTA, so CL times fewer instances are in flight and their
// positions and adjacency stay in L2 across the iterations).  The phases are
// separated by the hardware cluster barrier (release / acquire at cluster
// scope, so global writes of one CTA are visible to the others after it);
// the instance index and the cloth box live in the leader CTA's shared
// memory and are reached through distributed shared memory.
template <int CL>
__device__ __forceinline__ void inst_sync() {
    if constexpr (CL == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of `p` (this CTA's shared memory) in CTA `rank`
__device__ __forceinline__ unsigned leader_addr(const void* p, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r)
                 : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ int ld_cluster_s32(unsigned addr) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void red_cluster_min(unsigned addr, unsigned v) {
    asm volatile("red.shared::cluster.min.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void red_cluster_max(unsigned addr, unsigned v) {
    asm volatile("red.shared::cluster.max.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <int BLOCK, int MINB, int CL, bool FAST>
__global__ void __launch_bounds__(BLOCK, MINB) batched_substep_kernel(BatchedSubstepArgs A) {
    pdl_entry();
    constexpr int NW = BLOCK / 32;
    constexpr int STRIDE = CL * BLOCK;  // threads working on one instance
    constexpr int NWI = CL * NW;        // warps working on one instance
    __shared__ int s_inst;
    __shared__ unsigned s_box[6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned rank = CL == 1 ? 0u : cluster_rank();
    const int gtid = (int)rank * BLOCK + tid, gwarp = (int)rank * NW + warp;
    int bad = 0, overflow = 0;
    for (;;) {
        inst_sync<CL>();
        if (rank == 0) {
            if (tid == 0) {
                const int k = atomicAdd(A.queue, 1);
                s_inst = k < A.n_inst ? A.order[k] : -1;
            }
            if (tid < 6) s_box[tid] = tid < 3 ? f2ord_c(1e5f) : f2ord_c(-1e5f);
        }
        inst_sync<CL>();
        const int i = CL == 1 ? s_inst : ld_cluster_s32(leader_addr(&s_inst, 0));
        if (i < 0) break;
        const int v0 = A.vptr[i], v1 = A.vptr[i + 1], f0 = A.fptr[i], f1 = A.fptr[i + 1], c0 = A.cptr[i];
        const int o0 = A.optr[i], o1 = A.optr[i + 1];
        // the cloth box on x (segment_aabb_kernel) ...
        {
            float lo[3] = {1e5f, 1e5f, 1e5f}, hi[3] = {-1e5f, -1e5f, -1e5f};
            for (int v = v0 + gtid; v < v1; v += STRIDE) {
                const float4 p = A.x4[v];
                lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
                hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
            }
            for (int k = 0; k < 3; ++k) {
                for (int o = 16; o > 0; o >>= 1) {
                    lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                    hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
                }
            }
            if (lane == 0) {
                for (int k = 0; k < 3; ++k) {
                    if (CL == 1) {
                        atomicMin(s_box + k, f2ord_c(lo[k]));
                        atomicMax(s_box + 3 + k, f2ord_c(hi[k]));
                    } else {
                        red_cluster_min(leader_addr(s_box + k, 0), f2ord_c(lo[k]));
                        red_cluster_max(leader_addr(s_box + 3 + k, 0), f2ord_c(hi[k]));
                    }
                }
            }
        }
        // ... padded face boxes on x (face_aabb_kernel) and the unions of
        // chunks of 32 of them (warp w of a pass: chunk w)
        for (int fb = f0 + 32 * gwarp; fb < f1; fb += 32 * NWI) {
            const int f = fb + lane;
            V3 lo{INFINITY, INFINITY, INFINITY}, hi{-INFINITY, -INFINITY, -INFINITY};
            if (f < f1) {
                const V3 a = mk(A.x4[A.faces[3 * f]]), b = mk(A.x4[A.faces[3 * f + 1]]),
                         c = mk(A.x4[A.faces[3 * f + 2]]);
                const V3 l = vmin(vmin(a, b), c), h = vmax(vmax(a, b), c);
                lo = V3{l.x - A.pad, l.y - A.pad, l.z - A.pad};
                hi = V3{h.x + A.pad, h.y + A.pad, h.z + A.pad};
                A.fmin4[f] = make_float4(lo.x, lo.y, lo.z, 0.0f);
                A.fmax4[f] = make_float4(hi.x, hi.y, hi.z, 0.0f);
            }
            for (int o = 16; o > 0; o >>= 1) {
                lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
                lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
                lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
                hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
                hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
                hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
            }
            if (lane == 0) {
                const int c = c0 + (fb - f0) / 32;
                A.cmin4[c] = make_float4(lo.x, lo.y, lo.z, 0.0f);
                A.cmax4[c] = make_float4(hi.x, hi.y, hi.z, 0.0f);
            }
        }
        // compute_y (predict_kernel)
        if (A.predict) {
            for (int v = v0 + gtid; v < v1; v += STRIDE) {
                const float4 x = A.x4[v], vel = A.v4[v];
                const float f = A.fixed[v];
                float4 y;
                y.x = (x.x + (f * vel.x) * A.dt) + (A.gx * A.dt) * A.dt;
                y.y = (x.y + (f * vel.y) * A.dt) + (A.gy * A.dt) * A.dt;
                y.z = (x.z + (f * vel.z) * A.dt) + (A.gz * A.dt) * A.dt;
                y.w = x.w;
                A.ya[v] = y;
            }
        }
        inst_sync<CL>();
        if (rank == 0 && tid < 6) {
            const float b = ord2f_c(s_box[tid]);
            A.cl_box6[6 * i + tid] = tid < 3 ? b - A.pad : b + A.pad;
        }
        float4* yin = A.ya;
        float4* yout = A.yb;
        for (int it = 0; it < A.n_iter; ++it) {
            if (A.nbr16 != nullptr) {
                for (int v = v0 + gtid; v < v1; v += STRIDE)
                    yout[v] = sweep_vertex_src<2, true, FAST, false, false>(
                        v, A.x4, yin, A.fixed, __ldg(A.adj_ptr + v), __ldg(A.adj_ptr + v + 1),
                        AdjPacked{A.nbr16, A.rest32, 0}, A.ks, A.kb, 1, nullptr);
            } else {
                for (int v = v0 + gtid; v < v1; v += STRIDE)
                    yout[v] = sweep_vertex<2, true, FAST, false, false>(v, A.x4, yin, A.fixed, A.adj_ptr, A.adj,
                                                                        A.ks, A.kb, 1, nullptr);
            }
            inst_sync<CL>();
            if (it == 0) {
                // broad phase (batched_vt_st_broad_kernel, batched_tv_st_broad_kernel)
                const int of0 = A.ob_fptr[i], of1 = A.ob_fptr[i + 1];
                const float* ob6 = A.ob_box6 + 6 * i;
                for (int v = v0 + gtid; v < v1; v += STRIDE) {
                    const V3 p = mk(yout[v]);
                    const V3 a{p.x - A.pad, p.y - A.pad, p.z - A.pad}, b{p.x + A.pad, p.y + A.pad, p.z + A.pad};
                    unsigned m = 0;
                    if (!query_skipped(a, b, ob6))
                        for (int f = of0; f < of1; ++f)
                            if (overlap(a, b, mk(A.ob_fmin4[f]), mk(A.ob_fmax4[f]))) m |= 1u << (f - of0);
                    A.vmask[v] = m;
                }
                const float* cb6 = A.cl_box6 + 6 * i;
                const int nch = (f1 - f0 + 31) / 32;
                for (int s = o0 + gwarp; s < o1; s += NWI) {
                    const V3 p = mk(A.xs4[s]);
                    const V3 a{p.x - A.pad, p.y - A.pad, p.z - A.pad}, b{p.x + A.pad, p.y + A.pad, p.z + A.pad};
                    int count = 0;
                    if (!query_skipped(a, b, cb6)) {
                        for (int cb = 0; cb < nch; cb += 32) {
                            const int c = cb + lane;
                            const bool near_ = c < nch && overlap(a, b, mk(A.cmin4[c0 + c]), mk(A.cmax4[c0 + c]));
                            unsigned hits = __ballot_sync(0xffffffffu, near_);
                            while (hits) {
                                const int ch = cb + __ffs(hits) - 1;
                                hits &= hits - 1u;
                                const int f = f0 + 32 * ch + lane;
                                const bool hit = f < f1 && overlap(a, b, mk(A.fmin4[f]), mk(A.fmax4[f]));
                                const unsigned ball = __ballot_sync(0xffffffffu, hit);
                                const int slot = count + __popc(ball & ((1u << lane) - 1u));
                                if (hit && slot < A.cap) A.tv_cand[(size_t)s * A.cap + slot] = f;
                                count += __popc(ball);
                            }
                        }
                    }
                    if (lane == 0) {
                        A.tv_num[s] = count;
                        if (count > A.cap) overflow = 1;
                    }
                }
                inst_sync<CL>();
            }
            // obstacle contacts (batched_contacts_kernel)
            const int nv = v1 - v0;
            for (int k = gtid; k < nv + (o1 - o0); k += STRIDE) {
                if (k < nv) {
                    const int v = v0 + k;
                    unsigned m = A.vmask[v];
                    if (m) {
                        const int of0 = A.ob_fptr[i];
                        const V3 x0 = mk(yout[v]);
                        while (m) {
                            const int kk = __ffs(m) - 1;
                            m &= m - 1;
                            const int f = of0 + kk;
                            const V3 x[4] = {x0, mk(A.xs4[A.ob_faces[3 * f]]), mk(A.xs4[A.ob_faces[3 * f + 1]]),
                                             mk(A.xs4[A.ob_faces[3 * f + 2]])};
                            pair_project_lean(VT_ST, make_int4(v, -1, -1, -1), x, A.fixed, A.m_inv, A.dHat,
                                              A.compliance, A.dx, A.nc, &bad);
                        }
                    }
                } else {
                    const int s = o0 + (k - nv);
                    const int n = min(A.tv_num[s], A.cap);
                    for (int j = 0; j < n; ++j) {
                        const int fd = A.tv_cand[(size_t)s * A.cap + j];
                        const int4 vv = make_int4(-1, A.faces[3 * fd], A.faces[3 * fd + 1], A.faces[3 * fd + 2]);
                        const V3 x[4] = {mk(A.xs4[s]), mk(yout[vv.y]), mk(yout[vv.z]), mk(yout[vv.w])};
                        pair_project_lean(TV_ST, vv, x, A.fixed, A.m_inv, A.dHat, A.compliance, A.dx, A.nc, &bad);
                    }
                }
            }
            inst_sync<CL>();
            // update_dx (collision_apply_kernel)
            for (int v = v0 + gtid; v < v1; v += STRIDE) {
                const int c = A.nc[v];
                if (c > 0) {
                    const float cf = (float)c;
                    const float f = A.fixed[v];
                    float4 y = yout[v];
                    y.x = y.x + f * (from_fix(A.dx[3 * v]) / cf);
                    y.y = y.y + f * (from_fix(A.dx[3 * v + 1]) / cf);
                    y.z = y.z + f * (from_fix(A.dx[3 * v + 2]) / cf);
                    yout[v] = y;
                    A.dx[3 * v] = 0;
                    A.dx[3 * v + 1] = 0;
                    A.dx[3 * v + 2] = 0;
                    A.nc[v] = 0;
                }
            }
            inst_sync<CL>();
            float4* t = yin;
            yin = yout;
            yout = t;
        }
        // compute_velocity + update_x (velocity_update_kernel) from the final y
        for (int v = v0 + gtid; v < v1; v += STRIDE) {
            float4 x = A.x4[v];
            const float4 y = yin[v];
            const float sfac = (1.0f - A.damping) * A.fixed[v];
            float4 vel;
            vel.x = (sfac * (y.x - x.x)) / A.dt;
            vel.y = (sfac * (y.y - x.y)) / A.dt;
            vel.z = (sfac * (y.z - x.z)) / A.dt;
            vel.w = 0.0f;
            A.v4[v] = vel;
            x.x = x.x + A.dt * vel.x;
            x.y = x.y + A.dt * vel.y;
            x.z = x.z + A.dt * vel.z;
            A.x4[v] = x;
        }
    }
    // no CTA leaves while another CTA of its cluster may still read its
    // shared memory (the final instance index)
    if (CL > 1) inst_sync<CL>();
    if (bad) atomicOr(A.status, SX_STATUS_FIXED_RANGE);
    if (overflow) atomicOr(A.status, SX_STATUS_CAND_OVERFLOW);
    // the last CTA out resets the queue for the next launch
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(A.queue + 1, 1) == (int)gridDim.x - 1) {
            A.queue[0] = 0;
            A.queue[1] = 0;
        }
    }
}

// ---------------------------------------------------------------------------
// Velocity-level contact and friction (solve_constraints_v, XPBD.py:374-381
// and :398-404; collision_constraints_v.py __vt_st :6-133, __tv_st :137-330,
// __vt_dy :334-570), over the pair records of the last position-level contact
// sweep (pair, g, schur).  For a record with Cv = sum g_k . v_k < 0: a normal
// velocity impulse, then a tangential one towards the feature's (weighted)
// velocity, scaled by mu unless mu |Cv| > cTan.  Each `dv += ...` pairs with
// `nc += 1`; dv is accumulated in fixed point (order independent) and applied
// as v += fixed * dv / nc where m_inv > 0 (update_dv).  Written in the
// reference's evaluation order, including its quirks: __vt_st region 3 scales
// the normal impulse by the static mesh's m_inv indexed by the dynamic vertex
// id (0 where that id is past the static mesh), region 5 reverses the
// tangential direction; __tv_st's Cv weights v2 with g3; __vt_dy region 1
// scales the second vertex's tangential impulse by m_inv of v1.
// ---------------------------------------------------------------------------
__device__ __forceinline__ V3 vmul(V3 a, float s) { return V3{a.x * s, a.y * s, a.z * s}; }  // (v * s)
__device__ __forceinline__ float vnorm(V3 a) { return sqrtf(dot(a, a)); }

struct VelCtx {
    const float4* v4;
    const float4* vs4;
    const float* fixed;
    const float* m_inv;
    const float* m_inv_st;
    int Vs;
    long long* dv;
    int* nc;
    int* bad;
};
__device__ __forceinline__ V3 vel(const VelCtx& c, int v) { return mk(c.v4[v]); }
__device__ __forceinline__ V3 vel_st(const VelCtx& c, int v) { return mk(c.vs4[v]); }
__device__ __forceinline__ void dv_add(const VelCtx& c, int v, V3 d) {
    acc_add(c.dv, c.nc, v, 1.0f, d, c.bad);  // 1.0f * d is exact
}

// static triangle (v1..v3) vs dynamic vertex v0 (collision_constraints_v.py:6-133)
__device__ void vel_vt_st(const VelCtx& c, int v0, int v1, int v2, int v3, int dtype, const V3 g[4], float schur,
                          float mu) {
    const V3 u0 = vel(c, v0), u1 = vel_st(c, v1), u2 = vel_st(c, v2), u3 = vel_st(c, v3);
    const float Cv = ((dot(g[0], u0) + dot(g[1], u1)) + dot(g[2], u2)) + dot(g[3], u3);
    if (!(Cv < 0.0f) || dtype < 0 || dtype > 6) return;
    const float ld_v = -Cv / schur;
    const float m0 = c.m_inv[v0];
    const float mn = dtype == 3 ? (v0 < c.Vs ? c.m_inv_st[v0] : 0.0f) : m0;
    dv_add(c, v0, scale(mn * ld_v, g[0]));
    const V3 vTan0 = add(u0, scale(m0 * ld_v, g[0]));
    V3 p;
    if (dtype <= 2) {
        p = dtype == 0 ? u1 : dtype == 1 ? u2 : u3;
    } else if (dtype == 6) {
        const float a = vnorm(g[1]), b = vnorm(g[2]), d = vnorm(g[3]);
        const float s = (a + b) + d;
        p = V3{((a * u1.x + b * u2.x) + d * u3.x) / s, ((a * u1.y + b * u2.y) + d * u3.y) / s,
               ((a * u1.z + b * u2.z) + d * u3.z) / s};
    } else {
        const V3 ua = dtype == 4 ? u2 : u1, ub = dtype == 3 ? u2 : u3;
        const float a = vnorm(dtype == 4 ? g[2] : g[1]), b = vnorm(dtype == 3 ? g[2] : g[3]);
        const float s = a + b;
        p = V3{(a * ua.x + b * ub.x) / s, (a * ua.y + b * ub.y) / s, (a * ua.z + b * ub.z) / s};
    }
    const V3 g0Tan = dtype == 5 ? sub(vTan0, p) : sub(p, vTan0);
    const float cTan = 0.5f * dot(g0Tan, g0Tan);
    const float sT = m0 * dot(g0Tan, g0Tan) + 1e-4f;
    const float ldTan = cTan / sT;
    const V3 dvTan = scale(m0 * ldTan, g0Tan);
    const float mu_e = mu * fabsf(Cv) > cTan ? 1.0f : mu;
    dv_add(c, v0, scale(mu_e, dvTan));
}

// static vertex v0 vs dynamic triangle (v1..v3) (collision_constraints_v.py:137-330)
__device__ void vel_tv_st(const VelCtx& c, int v0, const int vt[3], int dtype, const V3 g[4], float schur,
                          float mu) {
    const V3 w0 = vel_st(c, v0);
    const V3 u[3] = {vel(c, vt[0]), vel(c, vt[1]), vel(c, vt[2])};
    const float Cv = ((dot(g[0], w0) + dot(g[1], u[0])) + dot(g[3], u[1])) + dot(g[3], u[2]);
    if (!(Cv < 0.0f) || dtype < 0 || dtype > 6) return;
    const float ld_v = -Cv / schur;
    // participating triangle corners (index into vt/u, gradient index = k + 1)
    int ks[3], n;
    if (dtype <= 2) { ks[0] = dtype; n = 1; }
    else if (dtype == 3) { ks[0] = 0; ks[1] = 1; n = 2; }
    else if (dtype == 4) { ks[0] = 1; ks[1] = 2; n = 2; }
    else if (dtype == 5) { ks[0] = 0; ks[1] = 2; n = 2; }
    else { ks[0] = 0; ks[1] = 1; ks[2] = 2; n = 3; }
    V3 vTan[3];
    float m[3];
    for (int i = 0; i < n; ++i) {
        const int k = ks[i], vid = vt[k];
        const float fm = c.fixed[vid] * c.m_inv[vid];
        m[i] = c.m_inv[vid];
        dv_add(c, vid, scale(fm * ld_v, g[k + 1]));
        vTan[i] = add(u[k], vmul(scale(fm, g[k + 1]), ld_v));
    }
    if (n == 1) {
        const V3 gT = sub(w0, vTan[0]);
        const float cTan = 0.5f * dot(gT, gT);
        const float sT = m[0] * dot(gT, gT) + 1e-4f;
        const float ldTan = cTan / sT;
        const float mu_e = mu * fabsf(Cv) > cTan ? 1.0f : mu;
        dv_add(c, vt[ks[0]], scale(mu_e, scale(m[0] * ldTan, gT)));
        return;
    }
    float w[3], s;
    V3 p;
    if (n == 2) {
        w[0] = vnorm(g[ks[0] + 1]);
        w[1] = vnorm(g[ks[1] + 1]);
        s = w[0] + w[1];
        p = V3{(w[0] * vTan[0].x + w[1] * vTan[1].x) / s, (w[0] * vTan[0].y + w[1] * vTan[1].y) / s,
               (w[0] * vTan[0].z + w[1] * vTan[1].z) / s};
    } else {
        w[0] = vnorm(g[1]);
        w[1] = vnorm(g[2]);
        w[2] = vnorm(g[3]);
        s = (w[0] + w[1]) + w[2];
        p = V3{((w[0] * vTan[0].x + w[1] * vTan[1].x) + w[2] * vTan[2].x) / s,
               ((w[0] * vTan[0].y + w[1] * vTan[1].y) + w[2] * vTan[2].y) / s,
               ((w[0] * vTan[0].z + w[1] * vTan[1].z) + w[2] * vTan[2].z) / s};
    }
    const V3 d = sub(w0, p);
    V3 gT[3];
    float sT = 0.0f;
    for (int i = 0; i < n; ++i) {
        gT[i] = scale(w[i] / s, d);
        const float t = m[i] * dot(gT[i], gT[i]);
        sT = i == 0 ? t : sT + t;
    }
    const float cTan = 0.5f * dot(d, d);
    sT = sT + 1e-4f;
    const float ldTan = cTan / sT;
    const float mu_e = mu * fabsf(Cv) > cTan ? 1.0f : mu;
    for (int i = 0; i < n; ++i) dv_add(c, vt[ks[i]], scale(mu_e, scale(m[i] * ldTan, gT[i])));
}

// self contact, all dynamic (collision_constraints_v.py:334-570)
__device__ void vel_vt_dy(const VelCtx& c, const int vv[4], int dtype, const V3 g[4], float schur, float mu) {
    const V3 u[4] = {vel(c, vv[0]), vel(c, vv[1]), vel(c, vv[2]), vel(c, vv[3])};
    const float Cv = ((dot(g[0], u[0]) + dot(g[1], u[1])) + dot(g[2], u[2])) + dot(g[3], u[3]);
    if (!(Cv < 0.0f) || dtype < 0 || dtype > 6) return;
    const float ld_v = -Cv / schur;
    // participants: the query vertex and the feature's corners (gradient index)
    int ks[4], n;
    ks[0] = 0;
    if (dtype <= 2) { ks[1] = dtype + 1; n = 2; }
    else if (dtype == 3) { ks[1] = 1; ks[2] = 2; n = 3; }
    else if (dtype == 4) { ks[1] = 2; ks[2] = 3; n = 3; }
    else if (dtype == 5) { ks[1] = 1; ks[2] = 3; n = 3; }
    else { ks[1] = 1; ks[2] = 2; ks[3] = 3; n = 4; }
    V3 vTan[4];
    for (int i = 0; i < n; ++i) {
        const int k = ks[i], vid = vv[k];
        const float fm = c.fixed[vid] * c.m_inv[vid];
        dv_add(c, vid, vmul(scale(fm, g[k]), ld_v));
        vTan[i] = add(u[k], vmul(scale(fm, g[k]), ld_v));
    }
    V3 gT[4];
    float cTan, sT;
    if (n == 2) {
        gT[0] = neg(sub(vTan[0], vTan[1]));
        gT[1] = sub(vTan[0], vTan[1]);
        cTan = 0.5f * (dot(gT[1], gT[1]) + dot(gT[0], gT[0]));
        sT = (c.m_inv[vv[0]] * dot(gT[0], gT[0]) + c.m_inv[vv[ks[1]]] * dot(gT[1], gT[1])) + 1e-4f;
    } else {
        float w[3], s;
        V3 p;
        if (n == 3) {
            w[0] = vnorm(g[ks[1]]);
            w[1] = vnorm(g[ks[2]]);
            s = w[0] + w[1];
            p = V3{(w[0] * vTan[1].x + w[1] * vTan[2].x) / s, (w[0] * vTan[1].y + w[1] * vTan[2].y) / s,
                   (w[0] * vTan[1].z + w[1] * vTan[2].z) / s};
        } else {
            w[0] = vnorm(g[1]);
            w[1] = vnorm(g[2]);
            w[2] = vnorm(g[3]);
            s = (w[0] + w[1]) + w[2];
            p = V3{((w[0] * vTan[1].x + w[1] * vTan[2].x) + w[2] * vTan[3].x) / s,
                   ((w[0] * vTan[1].y + w[1] * vTan[2].y) + w[2] * vTan[3].y) / s,
                   ((w[0] * vTan[1].z + w[1] * vTan[2].z) + w[2] * vTan[3].z) / s};
        }
        gT[0] = sub(p, vTan[0]);
        for (int i = 1; i < n; ++i) gT[i] = scale(-(w[i - 1] / s), gT[0]);
        cTan = dot(gT[0], gT[0]);
        sT = c.m_inv[vv[0]] * dot(gT[0], gT[0]);
        for (int i = 1; i < n; ++i) {
            cTan = cTan + dot(gT[i], gT[i]);
            sT = sT + c.m_inv[vv[ks[i]]] * dot(gT[i], gT[i]);
        }
        cTan = 0.5f * cTan;
        sT = sT + 1e-4f;
    }
    const float ldTan = cTan / sT;
    const float mu_e = mu * fabsf(Cv) > cTan ? 1.0f : mu;
    for (int i = 0; i < n; ++i) {
        // region 1 scales the second vertex's impulse by m_inv of v1 (collision_constraints_v.py:410)
        const int mv = (dtype == 1 && i == 1) ? vv[1] : vv[ks[i]];
        dv_add(c, vv[ks[i]], scale(mu_e, scale(c.m_inv[mv] * ldTan, gT[i])));
    }
}

__global__ void __launch_bounds__(128) velocity_contact_kernel(
    int Vd, int Vs, const int* __restrict__ faces_dy, const int* __restrict__ faces_st, int cap,
    const int* __restrict__ pair, const float4* __restrict__ pair_g, const float* __restrict__ pair_schur,
    const int* __restrict__ pair_num, const float4* __restrict__ v4, const float4* __restrict__ vs4,
    const float* __restrict__ fixed, const float* __restrict__ m_inv, const float* __restrict__ m_inv_st, float mu,
    long long* dv, int* nc, int* status) {
    pdl_entry();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 2 * Vd + Vs) return;
    int bad = 0;
    const VelCtx c{v4, vs4, fixed, m_inv, m_inv_st, Vs, dv, nc, &bad};
    const int n = min(pair_num[q], cap);
    for (int j = 0; j < n; ++j) {
        const size_t o = (size_t)q * cap + j;
        const int face = pair[2 * o], dtype = pair[2 * o + 1];
        const V3 g[4] = {mk(pair_g[4 * o]), mk(pair_g[4 * o + 1]), mk(pair_g[4 * o + 2]), mk(pair_g[4 * o + 3])};
        const float sc = pair_schur[o];
        if (q < Vd) {
            vel_vt_st(c, q, faces_st[3 * face], faces_st[3 * face + 1], faces_st[3 * face + 2], dtype, g, sc, mu);
        } else if (q < 2 * Vd) {
            const int vv[4] = {q - Vd, faces_dy[3 * face], faces_dy[3 * face + 1], faces_dy[3 * face + 2]};
            vel_vt_dy(c, vv, dtype, g, sc, mu);
        } else {
            const int vt[3] = {faces_dy[3 * face], faces_dy[3 * face + 1], faces_dy[3 * face + 2]};
            vel_tv_st(c, q - 2 * Vd, vt, dtype, g, sc, mu);
        }
    }
    if (bad) atomicOr(status, SX_STATUS_FIXED_RANGE);
}

// update_dv (XPBD.py:398-404): v += fixed * dv / nc where m_inv > 0; clears dv, nc
__global__ void velocity_apply_kernel(int V, float4* __restrict__ v4, const float* __restrict__ fixed,
                                      const float* __restrict__ m_inv, long long* __restrict__ dv,
                                      int* __restrict__ nc) {
    pdl_entry();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int cnt = nc[v];
    if (cnt > 0) {
        if (m_inv[v] > 0.0f) {
            const float cf = (float)cnt, f = fixed[v];
            float4 u = v4[v];
            u.x = u.x + f * (from_fix(dv[3 * v]) / cf);
            u.y = u.y + f * (from_fix(dv[3 * v + 1]) / cf);
            u.z = u.z + f * (from_fix(dv[3 * v + 2]) / cf);
            v4[v] = u;
        }
        dv[3 * v] = 0;
        dv[3 * v + 1] = 0;
        dv[3 * v + 2] = 0;
        nc[v] = 0;
    }
}

}  // namespace sx

using namespace sx;

extern "C" int sx_edge_edge_classify(int n, const float* p12, float dHat, int* dtype, float* d, float* g12,
                                     void* stream) {
    SX_REQUIRE(n >= 0, "sx_edge_edge_classify: n < 0");
    if (n == 0) return SX_OK;
    SX_REQUIRE(p12 && dtype && d && g12, "sx_edge_edge_classify: null pointer");
    launch(edge_edge_classify_kernel, grid_for(n, 128), 128, 0, as_stream(stream), n, p12, dHat, dtype, d, g12);
    return check_launch("edge_edge_classify_kernel");
}

extern "C" int sx_edge_edge_sweep(int n_edges_dy, const int* edges_dy, const int* edges_st, const int* face_edges_dy,
                                  const int* face_edges_st, const float* y4, const float* xs4, const float* fixed,
                                  const float* m_inv, float dHat, float compliance, int cap, const int* ee_st_cand,
                                  const int* ee_st_num, const int* ee_dy_cand, const int* ee_dy_num,
                                  long long* dx_fix, int* nc, int* pair, float* pair_g, float* pair_schur,
                                  int* pair_num, int* status, const int* conv, int iter, void* stream) {
    SX_REQUIRE(n_edges_dy >= 0 && cap >= 1, "sx_edge_edge_sweep: bad sizes");
    if (n_edges_dy == 0) return SX_OK;
    SX_REQUIRE(edges_dy && face_edges_dy && y4 && fixed && m_inv && ee_dy_cand && ee_dy_num && dx_fix && nc &&
                   status,
               "sx_edge_edge_sweep: null pointer");
    SX_REQUIRE(!ee_st_cand || (ee_st_num && edges_st && face_edges_st && xs4),
               "sx_edge_edge_sweep: null static-mesh pointer");
    SX_REQUIRE(!pair_num || (pair && pair_g && pair_schur), "sx_edge_edge_sweep: partial pair outputs");
    PairOut po{pair, pair_g, pair_schur, pair_num, cap};
    launch(edge_edge_kernel, grid_for(2LL * n_edges_dy, 128), 128, 0, as_stream(stream), n_edges_dy, edges_dy, edges_st, face_edges_dy, face_edges_st,
           (const float4*)y4, (const float4*)xs4, fixed, m_inv, dHat, compliance, cap, ee_st_cand, ee_st_num,
           ee_dy_cand, ee_dy_num, dx_fix, nc, po, status, conv, iter);
    return check_launch("edge_edge_kernel");
}

extern "C" int sx_collision_sweep(int n_dy, int n_st, const int* faces_dy, const int* faces_st, float* y4,
                                  const float* xs4, const float* fixed, const float* m_inv, float dHat,
                                  float compliance, int cap, const int* vt_st_cand, const int* vt_st_num,
                                  const int* vt_dy_cand, const int* vt_dy_num, const int* tv_st_cand,
                                  const int* tv_st_num, long long* dx_fix, int* nc, int* pair, float* pair_g,
                                  float* pair_schur, int* pair_num, int* status, void* stream) {
    SX_REQUIRE(n_dy >= 0 && n_st >= 0 && cap >= 1, "sx_collision_sweep: bad sizes");
    if (n_dy == 0) return SX_OK;
    SX_REQUIRE(faces_dy && y4 && fixed && m_inv && vt_dy_cand && vt_dy_num && dx_fix && nc && status,
               "sx_collision_sweep: null pointer");
    SX_REQUIRE(n_st == 0 || (faces_st && xs4 && vt_st_cand && vt_st_num && tv_st_cand && tv_st_num),
               "sx_collision_sweep: null static-mesh pointer");
    SX_REQUIRE(!pair_num || (pair && pair_g && pair_schur), "sx_collision_sweep: partial pair outputs");
    cudaStream_t s = as_stream(stream);
    PairOut po{pair, pair_g, pair_schur, pair_num, cap};
    const int total = 2 * n_dy + n_st;
    // with no static mesh the vt_st block has no candidates: point it at the
    // vt_dy block but force its counts to zero by passing n_st == 0 paths only
    const int* vsn = vt_st_num;
    const int* vsc = vt_st_cand;
    if (n_st == 0) {
        SX_REQUIRE(vt_st_num && vt_st_cand, "sx_collision_sweep: vt_st arrays required (may be zero counts)");
    }
    launch(collision_project_kernel, grid_for(total, 128), 128, 0, s, 
        n_dy, n_st, faces_dy, faces_st, (const float4*)y4, (const float4*)xs4, fixed, m_inv, dHat, compliance, cap,
        vsc, vsn, vt_dy_cand, vt_dy_num, tv_st_cand, tv_st_num, dx_fix, nc, po, status);
    int rc = check_launch("collision_project_kernel");
    if (rc) return rc;
    launch_apply(n_dy, (float4*)y4, fixed, dx_fix, nc, nullptr, 0, s);
    return check_launch("collision_apply_kernel");
}

static inline size_t a256(size_t b) { return (b + 255) & ~(size_t)255; }
static inline int pairs_blocks(int n_dy, int n_st) {
    return (2 * n_dy + n_st + 1 + PAIR_QUERIES - 1) / PAIR_QUERIES;
}

// workspace: [block totals][query totals][meta 64 ints]
struct PairsWs {
    int* block_tot;
    int* query_tot;
    int* meta;
    size_t bytes;
};
static PairsWs pairs_ws(void* ws, int n_dy, int n_st) {
    PairsWs w;
    char* p = (char*)ws;
    char* p0 = p;
    w.block_tot = (int*)p; p += a256((size_t)pairs_blocks(n_dy, n_st) * 4);
    w.query_tot = (int*)p; p += a256((2 * (size_t)n_dy + n_st) * 4);
    w.meta = (int*)p; p += 256;
    w.bytes = (size_t)(p - p0);
    return w;
}

extern "C" size_t sx_contact_pairs_workspace_bytes(int n_dy, int n_st) { return pairs_ws(nullptr, n_dy, n_st).bytes; }

extern "C" int sx_contact_pairs_build(int n_dy, int n_st, const int* faces_dy, const int* faces_st, int cap,
                                      const int* vt_st_cand, const int* vt_st_num, const int* vt_dy_cand,
                                      const int* vt_dy_num, const int* tv_st_cand, const int* tv_st_num, int* pairs,
                                      long long max_pairs, void* ws, size_t ws_bytes, void* stream) {
    SX_REQUIRE(n_dy >= 0 && n_st >= 0 && cap >= 1, "sx_contact_pairs_build: bad sizes");
    SX_REQUIRE(max_pairs >= (long long)(2 * n_dy + n_st) * cap,
               "sx_contact_pairs_build: pair buffer must hold (2*n_dy + n_st) * cap entries");
    SX_REQUIRE(ws && ws_bytes >= sx_contact_pairs_workspace_bytes(n_dy, n_st),
               "sx_contact_pairs_build: workspace too small");
    SX_REQUIRE(faces_dy && vt_st_cand && vt_st_num && vt_dy_cand && vt_dy_num && pairs,
               "sx_contact_pairs_build: null pointer");
    SX_REQUIRE(n_st == 0 || (faces_st && tv_st_cand && tv_st_num), "sx_contact_pairs_build: null static pointer");
    cudaStream_t s = as_stream(stream);
    const int nb = pairs_blocks(n_dy, n_st);
    PairsWs w = pairs_ws(ws, n_dy, n_st);
    launch(pairs_count_kernel, nb, PB, 0, s, n_dy, n_st, cap, faces_dy, vt_st_num, vt_dy_cand, vt_dy_num, tv_st_num,
           w.block_tot, w.query_tot);
    const int direct = nb <= PAIRS_DIRECT;
    if (!direct) launch(pairs_scan_kernel, 1, 1024, 0, s, nb, w.block_tot);
    launch(pairs_fill_kernel, nb, PB, 0, s, n_dy, n_st, cap, faces_dy, faces_st, vt_st_cand, vt_st_num, vt_dy_cand,
           vt_dy_num, tv_st_cand, tv_st_num, (const int*)w.block_tot, (const int*)w.query_tot, direct, (int4*)pairs,
           w.meta);
    return check_launch("sx_contact_pairs_build");
}

static int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            n = 132;
    }
    return n;
}

// Launch configurations of the pair projection: pair batches box-tested per
// warp step (U) and resident blocks per SM (the grid is that many blocks per
// SM; registers are capped to keep them resident).  All give identical
// results.  The default is the pipelined form with two pair batches per warp
// step and 3 blocks per SM (80 registers; at 64 the projection spills): us per
// launch for it / pipelined 1 x 4 / stacked 2 x 3 on the 64 x 64 box scene (63 K
// pairs) 4.7 / 5.4 / 6.3, a 181 x 139 sphere drape (74 K) 5.5 / 6.1 / 9.1, a 256
// x 256 one (1.43 M) 13.7 / 14.0 / 19.3.  With three copies of a branching
// narrow phase and FP64 fixed point the same launches took 7.8 / 9.8 / 19.0.
struct PairsProjectVariant {
    int unroll, blocks_per_sm, pipelined;
    decltype(&pairs_project_kernel<1, 4, false, false>) kern, headed;
};
#define SX_PAIRS_VARIANT(U, B, MINB, PIPE)                                                             \
    {U, B, PIPE ? 1 : 0, pairs_project_kernel<U, MINB, PIPE, false>,                                    \
     pairs_project_kernel<U, MINB, PIPE, PIPE>}  // the stacked form tests every pair
static const PairsProjectVariant kPairsProjectVariants[] = {
    SX_PAIRS_VARIANT(2, 3, 3, false), SX_PAIRS_VARIANT(1, 4, 4, false), SX_PAIRS_VARIANT(2, 6, 3, false),
    SX_PAIRS_VARIANT(4, 2, 2, false), SX_PAIRS_VARIANT(2, 3, 3, true),  SX_PAIRS_VARIANT(1, 4, 4, true),
    SX_PAIRS_VARIANT(2, 4, 4, true),
};
#undef SX_PAIRS_VARIANT
constexpr int kNumPairsProjectVariants = sizeof(kPairsProjectVariants) / sizeof(kPairsProjectVariants[0]);
constexpr int kPairsProjectDefault = 4;

extern "C" int sx_contact_pairs_project_variants(void) { return kNumPairsProjectVariants; }

extern "C" int sx_contact_pairs_project_variant_info(int variant, int* unroll, int* blocks_per_sm) {
    SX_REQUIRE(variant >= 0 && variant < kNumPairsProjectVariants && unroll && blocks_per_sm,
               "sx_contact_pairs_project_variant_info: bad variant");
    *unroll = kPairsProjectVariants[variant].unroll;
    *blocks_per_sm = kPairsProjectVariants[variant].blocks_per_sm;
    return SX_OK;
}

extern "C" int sx_contact_pairs_project_variant_pipelined(int variant) {
    SX_REQUIRE(variant >= 0 && variant < kNumPairsProjectVariants,
               "sx_contact_pairs_project_variant_pipelined: bad variant");
    return kPairsProjectVariants[variant].pipelined;
}

extern "C" int sx_contact_pairs_project_headed(int n_dy, int n_st, const int* pairs, const void* ws, const float* y4,
                                               const float* xs4, const float* fixed, const float* m_inv, float dHat,
                                               float compliance, float cull_d2, long long* dx_fix, int* nc,
                                               int* status, const int* conv, int iter, int variant, const int* heads,
                                               const unsigned* moved, void* stream) {
    SX_REQUIRE(variant >= 0 && variant < kNumPairsProjectVariants, "sx_contact_pairs_project_v: bad variant");
    SX_REQUIRE(n_dy >= 0 && n_st >= 0, "sx_contact_pairs_project: bad sizes");
    if (n_dy == 0) return SX_OK;
    SX_REQUIRE(pairs && ws && y4 && fixed && m_inv && dx_fix && nc && status,
               "sx_contact_pairs_project: null pointer");
    SX_REQUIRE(n_st == 0 || xs4, "sx_contact_pairs_project: null static positions");
    SX_REQUIRE(!heads == !moved && ((uintptr_t)heads & 15) == 0,
               "sx_contact_pairs_project_headed: heads (16-byte aligned) and moved go together");
    PairsWs w = pairs_ws(const_cast<void*>(ws), n_dy, n_st);
    const PairsProjectVariant& pv = kPairsProjectVariants[variant];
    // without a cull every pair is evaluated: the headed body has no such form
    launch(heads && cull_d2 > 0.0f ? pv.headed : pv.kern, sm_count() * pv.blocks_per_sm, PP_BLOCK, 0, as_stream(stream),
           (const int*)w.meta,
           (const int4*)pairs, (const float4*)y4, (const float4*)xs4, fixed, m_inv, dHat, compliance, cull_d2, dx_fix,
           nc, status, conv, iter, heads, moved);
    return check_launch("pairs_project_kernel");
}

extern "C" int sx_contact_pairs_project_v(int n_dy, int n_st, const int* pairs, const void* ws, const float* y4,
                                          const float* xs4, const float* fixed, const float* m_inv, float dHat,
                                          float compliance, float cull_d2, long long* dx_fix, int* nc, int* status,
                                          const int* conv, int iter, int variant, void* stream) {
    return sx_contact_pairs_project_headed(n_dy, n_st, pairs, ws, y4, xs4, fixed, m_inv, dHat, compliance, cull_d2,
                                           dx_fix, nc, status, conv, iter, variant, nullptr, nullptr, stream);
}

extern "C" int sx_contact_pairs_project(int n_dy, int n_st, const int* pairs, const void* ws, const float* y4,
                                        const float* xs4, const float* fixed, const float* m_inv, float dHat,
                                        float compliance, float cull_d2, long long* dx_fix, int* nc, int* status,
                                        const int* conv, int iter, void* stream) {
    return sx_contact_pairs_project_v(n_dy, n_st, pairs, ws, y4, xs4, fixed, m_inv, dHat, compliance, cull_d2, dx_fix,
                                      nc, status, conv, iter, kPairsProjectDefault, stream);
}

extern "C" int sx_contact_pairs_project_default_variant(void) { return kPairsProjectDefault; }

extern "C" size_t sx_contact_pairs_heads_bytes(int n_dy, int cap) {
    if (n_dy < 0 || cap < 1) return 0;
    return ((size_t)n_dy * cap + 31) / 32 * HEAD_WORDS * sizeof(int) + 16;
}

extern "C" int sx_contact_pairs_heads(int n_dy, int n_st, int cap, const int* pairs, void* ws, const float* y4,
                                      float cull_d2, int min_pairs, float* ref4, unsigned* moved, int* heads,
                                      size_t heads_bytes, void* stream) {
    SX_REQUIRE(n_dy >= 0 && n_st >= 0 && cap >= 1, "sx_contact_pairs_heads: bad sizes");
    if (n_dy == 0) return SX_OK;
    SX_REQUIRE(pairs && ws && y4 && ref4 && moved && heads, "sx_contact_pairs_heads: null pointer");
    SX_REQUIRE(((uintptr_t)heads & 15) == 0 && heads_bytes >= sx_contact_pairs_heads_bytes(n_dy, cap),
               "sx_contact_pairs_heads: heads must be 16-byte aligned and sx_contact_pairs_heads_bytes long");
    PairsWs w = pairs_ws(ws, n_dy, n_st);
    launch(pairs_heads_kernel, resident_blocks(pairs_heads_kernel, 256), 256, 0, as_stream(stream), n_dy, w.meta,
           (const int4*)pairs, (const float4*)y4, cull_d2, min_pairs, (float4*)ref4, moved, heads);
    return check_launch("pairs_heads_kernel");
}

extern "C" int sx_contact_apply(int n_dy, float* y4, const float* fixed, long long* dx_fix, int* nc, const int* conv,
                                int iter, void* stream) {
    SX_REQUIRE(n_dy >= 0, "sx_contact_apply: bad size");
    if (n_dy == 0) return SX_OK;
    SX_REQUIRE(y4 && fixed && dx_fix && nc, "sx_contact_apply: null pointer");
    launch_apply(n_dy, (float4*)y4, fixed, dx_fix, nc, conv, iter, as_stream(stream));
    return check_launch("collision_apply_kernel");
}

extern "C" int sx_contact_pairs_sweep(int n_dy, int n_st, const int* pairs, const void* ws, float* y4,
                                      const float* xs4, const float* fixed, const float* m_inv, float dHat,
                                      float compliance, float cull_d2, long long* dx_fix, int* nc, int* status,
                                      const int* conv, int iter, void* stream) {
    const int rc = sx_contact_pairs_project(n_dy, n_st, pairs, ws, y4, xs4, fixed, m_inv, dHat, compliance, cull_d2,
                                            dx_fix, nc, status, conv, iter, stream);
    if (rc) return rc;
    return sx_contact_apply(n_dy, y4, fixed, dx_fix, nc, conv, iter, stream);
}

extern "C" int sx_segment_aabbs(const float* p4, const int* seg_ptr, int n_seg, float padding, float* box6,
                                void* stream) {
    SX_REQUIRE(n_seg >= 0, "sx_segment_aabbs: n_seg < 0");
    if (n_seg == 0) return SX_OK;
    SX_REQUIRE(p4 && seg_ptr && box6, "sx_segment_aabbs: null pointer");
    launch(segment_aabb_kernel, n_seg, SEG_BLOCK, 0, as_stream(stream), (const float4*)p4, seg_ptr, padding, box6);
    return check_launch("segment_aabb_kernel");
}

extern "C" int sx_batched_obstacle_broadphase(int n_verts, const float* y4, const int* vinst, const float* ob_box6,
                                              const int* ob_fptr, const float* ob_fmin4, const float* ob_fmax4,
                                              float padding, unsigned* vmask, int n_ob_verts, const float* xs4,
                                              const int* svinst, const float* cl_box6, const int* cl_fptr,
                                              const float* cl_fmin4, const float* cl_fmax4, const float* cl_cmin4,
                                              const float* cl_cmax4, int cap, int* tv_cand, int* tv_num, int* status,
                                              void* stream) {
    SX_REQUIRE(n_verts >= 0 && n_ob_verts >= 0 && cap >= 1, "sx_batched_obstacle_broadphase: bad sizes");
    SX_REQUIRE(y4 && vinst && ob_box6 && ob_fptr && ob_fmin4 && ob_fmax4 && vmask && status,
               "sx_batched_obstacle_broadphase: null pointer");
    SX_REQUIRE(n_ob_verts == 0 || (xs4 && svinst && cl_box6 && cl_fptr && cl_fmin4 && cl_fmax4 && cl_cmin4 &&
                                   cl_cmax4 && tv_cand && tv_num),
               "sx_batched_obstacle_broadphase: null obstacle-vertex pointer");
    cudaStream_t s = as_stream(stream);
    if (n_verts > 0)
        launch(batched_vt_st_broad_kernel, grid_for(n_verts, 256), 256, 0, s, n_verts, (const float4*)y4, vinst,
               ob_box6, ob_fptr, (const float4*)ob_fmin4, (const float4*)ob_fmax4, padding, vmask);
    if (n_ob_verts > 0)
        launch(batched_tv_st_broad_kernel, grid_for(32LL * n_ob_verts, 256), 256, 0, s, n_ob_verts,
               (const float4*)xs4, svinst, cl_box6, cl_fptr, (const float4*)cl_fmin4, (const float4*)cl_fmax4,
               (const float4*)cl_cmin4, (const float4*)cl_cmax4, padding, cap, tv_cand, tv_num, status);
    return check_launch("sx_batched_obstacle_broadphase");
}

// list workspace: [count, 256 bytes][quads]
static long long list_capacity(int n_verts, int n_ob_verts, int cap) {
    return 8LL * n_verts + (long long)n_ob_verts * cap;
}

extern "C" size_t sx_batched_contact_list_bytes(int n_verts, int n_ob_verts, int cap) {
    if (n_verts < 0 || n_ob_verts < 0 || cap < 1) return 0;
    return 256 + (size_t)list_capacity(n_verts, n_ob_verts, cap) * sizeof(int4);
}

extern "C" int sx_batched_contact_list(int n_verts, const unsigned* vmask, const int* vinst, const int* ob_fptr,
                                       const int* ob_faces, int n_ob_verts, const int* tv_cand, const int* tv_num,
                                       int cap, const int* cl_faces, void* list, size_t list_bytes, void* stream) {
    SX_REQUIRE(n_verts >= 0 && n_ob_verts >= 0 && cap >= 1, "sx_batched_contact_list: bad sizes");
    SX_REQUIRE(list && ((uintptr_t)list & 15) == 0 &&
                   list_bytes >= sx_batched_contact_list_bytes(n_verts, n_ob_verts, cap),
               "sx_batched_contact_list: list must be 16-byte aligned and sx_batched_contact_list_bytes long");
    SX_REQUIRE(n_verts == 0 || (vmask && vinst && ob_fptr && ob_faces), "sx_batched_contact_list: null pointer");
    SX_REQUIRE(n_ob_verts == 0 || (tv_cand && tv_num && cl_faces), "sx_batched_contact_list: null pointer");
    cudaStream_t s = as_stream(stream);
    SX_CUDA(cudaMemsetAsync(list, 0, 256, s));
    const long long total = ((long long)n_verts + 31) / 32 * 32 + (long long)n_ob_verts * cap;
    if (total == 0) return SX_OK;
    launch(batched_list_kernel, grid_for(total, 256), 256, 0, s, n_verts, n_ob_verts, vmask, vinst, ob_fptr, ob_faces,
           tv_cand, tv_num, cap, cl_faces, (int4*)((char*)list + 256), list_capacity(n_verts, n_ob_verts, cap),
           (unsigned long long*)list);
    return check_launch("batched_list_kernel");
}

extern "C" int sx_batched_obstacle_contacts_listed(int n_verts, float* y4, const float* fixed, const float* m_inv,
                                                   const int* vinst, const int* ob_fptr, const int* ob_faces,
                                                   const float* xs4, const unsigned* vmask, int n_ob_verts,
                                                   const int* tv_cand, const int* tv_num, int cap,
                                                   const int* cl_faces, const void* list, float dHat,
                                                   float compliance, long long* dx_fix, int* nc, int* status,
                                                   const int* conv, int iter, void* stream) {
    SX_REQUIRE(n_verts >= 0 && n_ob_verts >= 0 && cap >= 1, "sx_batched_obstacle_contacts: bad sizes");
    if (n_verts == 0) return SX_OK;
    SX_REQUIRE(y4 && fixed && m_inv && vinst && ob_fptr && ob_faces && xs4 && vmask && dx_fix && nc && status,
               "sx_batched_obstacle_contacts: null pointer");
    SX_REQUIRE(n_ob_verts == 0 || (tv_cand && tv_num && cl_faces), "sx_batched_obstacle_contacts: null pointer");
    SX_REQUIRE(((uintptr_t)list & 15) == 0, "sx_batched_obstacle_contacts: list must be 16-byte aligned");
    cudaStream_t s = as_stream(stream);
    const long long tasks = ((long long)n_ob_verts * cap + 31) / 32 + ((long long)n_verts + 31) / 32;
    const long long full = (long long)sm_count() * BC_PER_SM, need = (tasks + BC_BLOCK / 32 - 1) / (BC_BLOCK / 32);
    launch(batched_contacts_kernel, (int)(need < full ? need : full), BC_BLOCK, 0, s, n_verts, n_ob_verts,
           (const float4*)y4, fixed, m_inv, vinst, ob_fptr, ob_faces, (const float4*)xs4, vmask, tv_cand, tv_num,
           cap, cl_faces, dHat, compliance, (const int4*)(list ? (const char*)list + 256 : nullptr),
           list_capacity(n_verts, n_ob_verts, cap), (const unsigned long long*)list, dx_fix, nc, status, conv, iter);
    int rc = check_launch("batched_contacts_kernel");
    if (rc) return rc;
    launch_apply(n_verts, (float4*)y4, fixed, dx_fix, nc, conv, iter, s);
    return check_launch("collision_apply_kernel");
}

extern "C" int sx_batched_obstacle_contacts(int n_verts, float* y4, const float* fixed, const float* m_inv,
                                            const int* vinst, const int* ob_fptr, const int* ob_faces,
                                            const float* xs4, const unsigned* vmask, int n_ob_verts,
                                            const int* tv_cand, const int* tv_num, int cap, const int* cl_faces,
                                            float dHat, float compliance, long long* dx_fix, int* nc, int* status,
                                            const int* conv, int iter, void* stream) {
    return sx_batched_obstacle_contacts_listed(n_verts, y4, fixed, m_inv, vinst, ob_fptr, ob_faces, xs4, vmask,
                                               n_ob_verts, tv_cand, tv_num, cap, cl_faces, nullptr, dHat, compliance,
                                               dx_fix, nc, status, conv, iter, stream);
}

// Launch configurations of the persistent batched substep: threads per CTA
// and CTAs per SM (the grid is that many per SM); all give identical results.
struct BatchedSubstepVariant {
    int block, blocks_per_sm, cluster;
    decltype(&batched_substep_kernel<256, 4, 1, false>) exact, fast;
};
#define SX_BS_VARIANT(B, M, CL) \
    {B, M, CL, batched_substep_kernel<B, M, CL, false>, batched_substep_kernel<B, M, CL, true>}
// (threads per CTA, CTAs per SM, CTAs per instance)
static const BatchedSubstepVariant kBatchedSubstepVariants[] = {
    SX_BS_VARIANT(512, 2, 1), SX_BS_VARIANT(256, 4, 1), SX_BS_VARIANT(1024, 1, 1), SX_BS_VARIANT(256, 2, 1),
    SX_BS_VARIANT(512, 1, 1), SX_BS_VARIANT(128, 8, 1), SX_BS_VARIANT(512, 2, 8), SX_BS_VARIANT(512, 2, 4),
    SX_BS_VARIANT(256, 4, 8), SX_BS_VARIANT(1024, 1, 8), SX_BS_VARIANT(512, 2, 2),
};
#undef SX_BS_VARIANT
constexpr int kNumBatchedSubstepVariants = sizeof(kBatchedSubstepVariants) / sizeof(kBatchedSubstepVariants[0]);

extern "C" int sx_batched_substep_variants(void) { return kNumBatchedSubstepVariants; }

extern "C" int sx_batched_substep_variant_info(int variant, int* block, int* blocks_per_sm) {
    SX_REQUIRE(variant >= 0 && variant < kNumBatchedSubstepVariants && block && blocks_per_sm,
               "sx_batched_substep_variant_info: bad variant");
    *block = kBatchedSubstepVariants[variant].block;
    *blocks_per_sm = kBatchedSubstepVariants[variant].blocks_per_sm;
    return SX_OK;
}

extern "C" int sx_batched_substep_variant_cluster(int variant) {
    SX_REQUIRE(variant >= 0 && variant < kNumBatchedSubstepVariants, "sx_batched_substep_variant_cluster: bad variant");
    return kBatchedSubstepVariants[variant].cluster;
}

extern "C" int sx_batched_substep(const SxBatchedSubstep* b, int variant, int fast, void* stream) {
    SX_REQUIRE(b, "sx_batched_substep: null argument block");
    SX_REQUIRE(variant >= 0 && variant < kNumBatchedSubstepVariants, "sx_batched_substep: bad variant");
    SX_REQUIRE(b->n_inst >= 0 && b->n_iter >= 0 && b->cap >= 1, "sx_batched_substep: bad sizes");
    if (b->n_inst == 0) return SX_OK;
    SX_REQUIRE(b->order && b->vptr && b->fptr && b->cptr && b->optr && b->ob_fptr && b->x4 && b->y4 && b->y_other4 &&
                   b->v4 && b->fixed && b->m_inv && b->adj_ptr && b->adj && b->faces && b->ob_faces && b->xs4 &&
                   b->fmin4 && b->fmax4 && b->cmin4 && b->cmax4 && b->cl_box6 && b->ob_box6 && b->ob_fmin4 &&
                   b->ob_fmax4 && b->vmask && b->tv_cand && b->tv_num && b->dx_fix && b->nc && b->status && b->queue,
               "sx_batched_substep: null pointer");
    BatchedSubstepArgs A;
    A.n_inst = b->n_inst; A.n_iter = b->n_iter; A.predict = b->predict; A.cap = b->cap;
    A.order = b->order; A.vptr = b->vptr; A.fptr = b->fptr; A.cptr = b->cptr; A.optr = b->optr;
    A.ob_fptr = b->ob_fptr;
    A.x4 = (float4*)b->x4; A.ya = (float4*)b->y4; A.yb = (float4*)b->y_other4; A.v4 = (float4*)b->v4;
    SX_REQUIRE((b->adj_nbr16 == nullptr) == (b->adj_rest32 == nullptr),
               "sx_batched_substep: give both packed adjacency arrays or neither");
    A.fixed = b->fixed; A.m_inv = b->m_inv; A.adj_ptr = b->adj_ptr; A.adj = (const int2*)b->adj;
    A.nbr16 = b->adj_nbr16; A.rest32 = b->adj_rest32;
    A.faces = b->faces; A.ob_faces = b->ob_faces; A.xs4 = (const float4*)b->xs4;
    A.fmin4 = (float4*)b->fmin4; A.fmax4 = (float4*)b->fmax4; A.cmin4 = (float4*)b->cmin4;
    A.cmax4 = (float4*)b->cmax4; A.cl_box6 = b->cl_box6; A.ob_box6 = b->ob_box6;
    A.ob_fmin4 = (const float4*)b->ob_fmin4; A.ob_fmax4 = (const float4*)b->ob_fmax4;
    A.vmask = b->vmask; A.tv_cand = b->tv_cand; A.tv_num = b->tv_num; A.dx = b->dx_fix; A.nc = b->nc;
    A.status = b->status; A.queue = b->queue;
    A.pad = b->padding; A.dt = b->dt; A.gx = b->gx; A.gy = b->gy; A.gz = b->gz; A.ks = b->k_spring;
    A.kb = b->k_bend; A.dHat = b->dHat; A.compliance = b->compliance; A.damping = b->damping;
    const BatchedSubstepVariant& bv = kBatchedSubstepVariants[variant];
    const auto kern = fast ? bv.fast : bv.exact;
    if (bv.cluster == 1) {
        launch(kern, sm_count() * bv.blocks_per_sm, bv.block, 0, as_stream(stream), A);
        return check_launch("batched_substep_kernel");
    }
    // clusters of bv.cluster CTAs, one instance per cluster
    const int clusters = max(1, sm_count() * bv.blocks_per_sm / bv.cluster);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * bv.cluster);
    cfg.blockDim = dim3(bv.block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = bv.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    int na = 1;
    if (pdl_enabled()) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        na = 2;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    SX_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
    note_launch();
    return check_launch("batched_substep_kernel");
}

extern "C" int sx_velocity_contacts(int n_dy, int n_st, const int* faces_dy, const int* faces_st, int cap,
                                    const int* pair, const float* pair_g, const float* pair_schur,
                                    const int* pair_num, float* v4, const float* vs4, const float* fixed,
                                    const float* m_inv, const float* m_inv_st, float mu, long long* dv_fix, int* nc,
                                    int* status, void* stream) {
    SX_REQUIRE(n_dy >= 0 && n_st >= 0 && cap >= 1, "sx_velocity_contacts: bad sizes");
    if (n_dy == 0) return SX_OK;
    SX_REQUIRE(faces_dy && pair && pair_g && pair_schur && pair_num && v4 && fixed && m_inv && dv_fix && nc && status,
               "sx_velocity_contacts: null pointer");
    SX_REQUIRE(n_st == 0 || (faces_st && vs4 && m_inv_st), "sx_velocity_contacts: null static pointer");
    cudaStream_t s = as_stream(stream);
    launch(velocity_contact_kernel, grid_for(2LL * n_dy + n_st, 128), 128, 0, s, n_dy, n_st, faces_dy, faces_st, cap,
           pair, (const float4*)pair_g, pair_schur, pair_num, (const float4*)v4, (const float4*)vs4, fixed, m_inv,
           m_inv_st, mu, dv_fix, nc, status);
    int rc = check_launch("velocity_contact_kernel");
    if (rc) return rc;
    launch(velocity_apply_kernel, grid_for(n_dy, 256), 256, 0, s, n_dy, (float4*)v4, fixed, m_inv, dv_fix, nc);
    return check_launch("velocity_apply_kernel");
}
