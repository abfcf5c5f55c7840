// One vertex of the Jacobi spring / bending sweep (XPBD.py:141-184 +
// :384-387), shared by the grid-wide sweep kernel and the persistent batched
// substep kernel so that both evaluate the same expressions in the same order.
//
// For a constraint (v0, v1) the reference computes x10 = p0 - p1,
// n = x10 * (1/|x10|), ld = k*C/(k*(w0+w1)*(n.n) + 1) and scatters
// dx0 -= (w0*ld)*n, dx1 += (w1*ld)*n with float atomics.  From v1's side
// p1 - p0 = -x10 exactly, so n flips sign exactly and
// dx1 - (w1*ld)*(-n) == dx1 + (w1*ld)*n bit for bit: every vertex evaluates
// dx -= (w_self*ld) * normalize(p_self - p_other) over its incident constraints
// in ascending constraint index, which equals a serial run of the reference.
//
// G: entries whose loads are issued together.  BY: bending pairs on y (the
// bend_y argument is then ignored).  FAST: fused multiply-adds, the hardware
// reciprocal square root, a fast divide and n.n taken as 1 (within float
// rounding of the exact form, not bit-identical).  CHECK: also sum C^2 into
// *c2.  YLDG: y is read through the read-only path (it does not change during
// the launch); kernels that write y themselves read it with plain loads.
#pragma once
#include "sx_common.cuh"
#include "sx_exact.cuh"

namespace sx {

template <bool YLDG>
__device__ __forceinline__ float4 load_y(const float4* p) {
    if (YLDG) return __ldg(p);
    return *p;
}

// Entry sources: entry k of vertex v's list as the adjacency word
// (neighbour | bit 31 for a bending pair, bits(rest length)).
struct AdjInt2 {  // the CSR of int2 entries
    const int2* __restrict__ adj;
    __device__ __forceinline__ int2 operator()(int, int k) const { return __ldg(adj + k); }
};
// The same entries read with the streaming (evict-first) cache policy: each
// entry is read once per sweep, so on a batch larger than L2 the positions,
// which neighbouring vertices gather again, keep their L2 lines.
struct AdjInt2Stream {
    const int2* __restrict__ adj;
    __device__ __forceinline__ int2 operator()(int, int k) const { return __ldcs(adj + k); }
};
// The packed CSR: nbr16[k] = neighbour - v, rest32[k] = bits(rest length) with
// bit 31 set for a bending pair (6 bytes per entry instead of 8), read from a
// shared-memory copy of the block's range [a0, a0 + n) when staged, else from
// global memory.
struct AdjPacked {
    const short* nbr;
    const unsigned* rest;
    int a0;
    __device__ __forceinline__ int2 operator()(int v, int k) const {
        const unsigned r = rest[k - a0];
        return make_int2((v + (int)nbr[k - a0]) | (int)(r & 0x80000000u), (int)(r & 0x7fffffffu));
    }
};

// The packed CSR read from global memory through the read-only path.
struct AdjPackedGlobal {
    const short* __restrict__ nbr;
    const unsigned* __restrict__ rest;
    __device__ __forceinline__ int2 operator()(int v, int k) const {
        const unsigned r = __ldg(rest + k);
        return make_int2((v + (int)__ldg(nbr + k)) | (int)(r & 0x80000000u), (int)(r & 0x7fffffffu));
    }
};

// One constraint from its owner's side: e = p_self - p_other, ws and wo the
// weights, kk the stiffness.  a0 * n is the term the owner subtracts (exact
// form); the fast form subtracts a0 * e.
//
// The exact form has two bodies with the same value: the straight-line one
// (sx_exact.cuh), which records the smallest and largest operand it met, and
// the one with '/' and sqrtf (IEEE), with which the caller evaluates the vertex
// again when they leave [2^-40, 2^40].  Inside it |e| and 1/|e| are safe, and C
// = |e| - rest is 0 or at least 2^-45 (the difference of two floats is a
// multiple of the smaller one's ulp), so that with 2^-20 <= |kk| <= 2^40 or
// kk = 0 (spring_k_ok) the numerator is 0 or at least 2^-65 and the quotient at
// least 2^-105.  (min and max pass over a NaN; both bodies then give NaN.)
// 1/|e| is its own reciprocal, not the square root's seed refined: that misses
// two significands in every other binade.
struct SpringTerm {
    float a0, x, y, z;
};
constexpr float kP2_40 = 1099511627776.0f;
struct SpringRange {
    float lo = 1.0f, hi = 1.0f;
    __device__ __forceinline__ bool ok() const { return lo >= 1.0f / kP2_40 && hi <= kP2_40; }
};

__device__ __forceinline__ bool spring_k_ok(float k) {
    return k == 0.0f || in_range(k, 1.0f / 1048576.0f, kP2_40);
}

template <bool FAST, bool IEEE>
__device__ __forceinline__ SpringTerm spring_term(float ex, float ey, float ez, float ws, float wo, float rest,
                                                  float kk, float* C, SpringRange* range) {
    if (FAST) {
        const float d2 = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, ez * ez));
        const float inv = rsqrtf(d2);
        *C = d2 * inv - rest;
        const float ld = __fdividef(kk * *C, __fmaf_rn(kk, ws + wo, 1.0f));
        return SpringTerm{(ws * ld) * inv, ex, ey, ez};  // times the unnormalised difference
    }
    const float d2 = (ex * ex + ey * ey) + ez * ez;
    const float lij = IEEE ? sqrtf(d2) : sqrt_rn(d2);
    *C = lij - rest;
    const float inv = IEEE ? 1.0f / lij : rcp_rn(lij);
    const float nx = inv * ex, ny = inv * ey, nz = inv * ez;
    const float schur = (ws + wo) * ((nx * nx + ny * ny) + nz * nz);
    const float num = kk * *C, den = kk * schur + 1.0f;
    if (!IEEE) {
        range->lo = fminf(fminf(range->lo, d2), den);
        range->hi = fmaxf(fmaxf(fmaxf(range->hi, d2), fabsf(num)), den);
    }
    const float ld = IEEE ? num / den : div_rn(num, den, rcp_rn(den));
    return SpringTerm{ws * ld, nx, ny, nz};
}

// y + fixed * (dx / nc) (update_dx, XPBD.py:384-387) for nc > 0 constraints
template <bool FAST, bool IEEE>
__device__ __forceinline__ float4 spring_update(float4 ps, float f, float dx, float dy, float dz, float nc, bool* ok) {
    float4 out = ps;
    if (FAST) {
        const float fs = __fdividef(f, nc);
        out.x = __fmaf_rn(fs, dx, ps.x);
        out.y = __fmaf_rn(fs, dy, ps.y);
        out.z = __fmaf_rn(fs, dz, ps.z);
    } else if (IEEE) {
        out.x = ps.x + f * (dx / nc);
        out.y = ps.y + f * (dy / nc);
        out.z = ps.z + f * (dz / nc);
    } else {
        // the sums never are -0 (they start at +0 and only subtract)
        const float r = rcp_rn(nc);
        out.x = ps.x + f * div_rn(dx, nc, r);
        out.y = ps.y + f * div_rn(dy, nc, r);
        out.z = ps.z + f * div_rn(dz, nc, r);
        constexpr float lo = 1.0f / (kP2_40 * kP2_40), hi = kP2_40 * kP2_40;
        *ok = *ok && (dx == 0.0f || in_range(dx, lo, hi)) && (dy == 0.0f || in_range(dy, lo, hi)) &&
              (dz == 0.0f || in_range(dz, lo, hi));
    }
    return out;
}

// G entries at a time, all their loads issued before the arithmetic, then the
// remaining ones singly.  The straight-line exact form also loads the next
// group's adjacency words beside this group's positions, so that a group waits
// for one round trip instead of two (PIPE).
template <int G, bool BY, bool FAST, bool CHECK, bool YLDG, bool IEEE, typename Src>
__device__ __forceinline__ float4 sweep_vertex_body(int v, float4 ps, const float4* __restrict__ x4, const float4* yin,
                                                    const float* __restrict__ fixed, int b, int e, const Src& src,
                                                    float ks, float kb, int bend_y, float* c2, bool* ok) {
    constexpr bool PIPE = !FAST && !IEEE;
    const float4 xs = BY ? ps : __ldg(x4 + v);
    float dx = 0.0f, dy = 0.0f, dz = 0.0f, sum2 = 0.0f;
    SpringRange range;
    auto load_o = [&](int2 a) {
        const bool use_x = !BY && a.x < 0 && !bend_y;
        const int u = a.x & 0x7fffffff;
        return use_x ? __ldg(x4 + u) : load_y<YLDG>(yin + u);
    };
    auto add_term = [&](int2 a, float4 o) {
        const bool bend = a.x < 0;
        const float4 self = !BY && bend && !bend_y ? xs : ps;
        float C;
        const SpringTerm t = spring_term<FAST, IEEE>(self.x - o.x, self.y - o.y, self.z - o.z, self.w, o.w,
                                                     __int_as_float(a.y), bend ? kb : ks, &C, &range);
        if (CHECK) sum2 = FAST ? __fmaf_rn(C, C, sum2) : sum2 + C * C;
        if (FAST) {
            dx = __fmaf_rn(-t.a0, t.x, dx);
            dy = __fmaf_rn(-t.a0, t.y, dy);
            dz = __fmaf_rn(-t.a0, t.z, dz);
        } else {
            dx = dx - t.a0 * t.x;
            dy = dy - t.a0 * t.y;
            dz = dz - t.a0 * t.z;
        }
    };
    int k0 = b;
    if (PIPE) {
        int2 a[G];
#pragma unroll
        for (int g = 0; g < G; ++g) a[g] = b + g < e ? src(v, b + g) : make_int2(0, 0);
        for (; k0 + G <= e; k0 += G) {
            int2 nx[G];
            float4 o[G];
#pragma unroll
            for (int g = 0; g < G; ++g) o[g] = load_o(a[g]);
#pragma unroll
            for (int g = 0; g < G; ++g) nx[g] = k0 + G + g < e ? src(v, k0 + G + g) : make_int2(0, 0);
#pragma unroll
            for (int g = 0; g < G; ++g) add_term(a[g], o[g]);
#pragma unroll
            for (int g = 0; g < G; ++g) a[g] = nx[g];
        }
        if (G > 1) {
#pragma unroll
            for (int g = 0; g < G - 1; ++g)
                if (k0 + g < e) add_term(a[g], load_o(a[g]));
        }
    } else {
        for (; k0 < e; k0 += G) {
            int2 a[G];
            float4 o[G];
#pragma unroll
            for (int g = 0; g < G; ++g) a[g] = k0 + g < e ? src(v, k0 + g) : make_int2(0, 0);
#pragma unroll
            for (int g = 0; g < G; ++g) o[g] = k0 + g < e ? load_o(a[g]) : ps;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (k0 + g >= e) break;
                add_term(a[g], o[g]);
            }
        }
    }
    if (CHECK) *c2 = sum2;
    if (e <= b) return ps;
    *ok = *ok && range.ok();
    return spring_update<FAST, IEEE>(ps, fixed[v], dx, dy, dz, (float)(e - b), ok);
}

// *c2 (CHECK): the vertex's sum of C^2
template <int G, bool BY, bool FAST, bool CHECK, bool YLDG, typename Src>
__device__ __forceinline__ float4 sweep_vertex_src(int v, const float4* __restrict__ x4, const float4* yin,
                                                   const float* __restrict__ fixed, int b, int e, const Src& src,
                                                   float ks, float kb, int bend_y, float* c2) {
    const float4 ps = load_y<YLDG>(yin + v);
    bool ok = FAST || (spring_k_ok(ks) && spring_k_ok(kb));
    float4 out = sweep_vertex_body<G, BY, FAST, CHECK, YLDG, false>(v, ps, x4, yin, fixed, b, e, src, ks, kb, bend_y,
                                                                    c2, &ok);
    if (!FAST && !ok)
        out = sweep_vertex_body<1, BY, FAST, CHECK, YLDG, true>(v, ps, x4, yin, fixed, b, e, src, ks, kb, bend_y, c2,
                                                                &ok);
    return out;
}

// The same vertex evaluated by L consecutive lanes of a warp (L = 2, 4 or 8).
// Lane j of the group evaluates entries b + j, b + j + L, ... (G of them per
// batch, loads issued together), and the group then adds the terms in
// ascending entry order, each lane receiving every term through shuffles, so
// each lane holds exactly the sums of sweep_vertex_src (same operations, same
// order).  A mesh with few vertices per SM keeps L times more loads in flight.
// Every lane of the warp must call it (a lane past the last vertex passes
// valid == false and b == e); the trip count is the warp's largest.
template <int L, int G, bool BY, bool FAST, bool YLDG, bool IEEE>
__device__ __forceinline__ float4 sweep_lanes_body(int v, bool valid, float4 ps, const float4* __restrict__ x4,
                                                   const float4* yin, const float* __restrict__ fixed, int b, int e,
                                                   const int2* __restrict__ adj, float ks, float kb, int bend_y,
                                                   bool* ok) {
    const int sub = threadIdx.x & (L - 1);
    const float4 xs = !BY && valid && e > b ? __ldg(x4 + v) : ps;
    float dx = 0.0f, dy = 0.0f, dz = 0.0f;
    SpringRange range;
    constexpr int SPAN = G * L;
    // stands in for a neighbour past the list's end: its term is in range and unused
    const float4 spare = make_float4(ps.x + 1.0f, ps.y, ps.z, 0.0f);
    const int steps = __reduce_max_sync(0xffffffffu, (e - b + SPAN - 1) / SPAN);
    for (int st = 0; st < steps; ++st) {
        const int k0 = b + st * SPAN;
        int2 a[G];
        float4 o[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int k = k0 + g * L + sub;
            a[g] = k < e ? __ldg(adj + k) : make_int2(0, 0);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int k = k0 + g * L + sub;
            const bool use_x = !BY && a[g].x < 0 && !bend_y;
            const int u = a[g].x & 0x7fffffff;
            o[g] = k < e ? (use_x ? __ldg(x4 + u) : load_y<YLDG>(yin + u)) : spare;
        }
        // per entry: exact form (a0 nx, a0 ny, a0 nz); fast form (a0, ex, ey, ez)
        float t0[G], t1[G], t2[G], t3[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const bool bend = a[g].x < 0;
            const float4 self = !BY && bend && !bend_y ? xs : ps;
            float C;
            const SpringTerm t = spring_term<FAST, IEEE>(self.x - o[g].x, self.y - o[g].y, self.z - o[g].z,
                                                         self.w, o[g].w, __int_as_float(a[g].y), bend ? kb : ks, &C,
                                                         &range);
            t0[g] = FAST ? t.a0 : t.a0 * t.x;
            t1[g] = FAST ? t.x : t.a0 * t.y;
            t2[g] = FAST ? t.y : t.a0 * t.z;
            t3[g] = FAST ? t.z : 0.0f;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int j = 0; j < L; ++j) {
                const int k = k0 + g * L + j;  // the same for every lane of the group
                const float q0 = __shfl_sync(0xffffffffu, t0[g], j, L);
                const float q1 = __shfl_sync(0xffffffffu, t1[g], j, L);
                const float q2 = __shfl_sync(0xffffffffu, t2[g], j, L);
                if (FAST) {
                    const float q3 = __shfl_sync(0xffffffffu, t3[g], j, L);
                    if (k < e) {
                        dx = __fmaf_rn(-q0, q1, dx);
                        dy = __fmaf_rn(-q0, q2, dy);
                        dz = __fmaf_rn(-q0, q3, dz);
                    }
                } else if (k < e) {
                    dx = dx - q0;
                    dy = dy - q1;
                    dz = dz - q2;
                }
            }
        }
    }
    if (e <= b) return ps;
    *ok = *ok && range.ok();
    return spring_update<FAST, IEEE>(ps, fixed[v], dx, dy, dz, (float)(e - b), ok);
}

// One lane of the warp out of range makes the whole warp evaluate its vertices
// again with the compiler's operations (the terms travel through shuffles).
template <int L, int G, bool BY, bool FAST, bool YLDG>
__device__ __forceinline__ float4 sweep_vertex_lanes(int v, bool valid, const float4* __restrict__ x4,
                                                     const float4* yin, const float* __restrict__ fixed, int b, int e,
                                                     const int2* __restrict__ adj, float ks, float kb, int bend_y) {
    static_assert(L == 2 || L == 4 || L == 8, "lanes per vertex: 2, 4 or 8");
    const float4 ps = valid ? load_y<YLDG>(yin + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    bool ok = FAST || (spring_k_ok(ks) && spring_k_ok(kb));
    float4 out =
        sweep_lanes_body<L, G, BY, FAST, YLDG, false>(v, valid, ps, x4, yin, fixed, b, e, adj, ks, kb, bend_y, &ok);
    if (!FAST && !__all_sync(0xffffffffu, ok))
        out = sweep_lanes_body<L, 1, BY, FAST, YLDG, true>(v, valid, ps, x4, yin, fixed, b, e, adj, ks, kb, bend_y,
                                                           &ok);
    return out;
}

template <int G, bool BY, bool FAST, bool CHECK, bool YLDG>
__device__ __forceinline__ float4 sweep_vertex(int v, const float4* __restrict__ x4, const float4* yin,
                                               const float* __restrict__ fixed, const int* __restrict__ ptr,
                                               const int2* __restrict__ adj, float ks, float kb, int bend_y,
                                               float* c2) {
    return sweep_vertex_src<G, BY, FAST, CHECK, YLDG>(v, x4, yin, fixed, __ldg(ptr + v), __ldg(ptr + v + 1),
                                                      AdjInt2{adj}, ks, kb, bend_y, c2);
}

// Motion of the vertices since a reference: the largest squared displacement of
// each block of 32 vertices, as float bits in moved[], raised by every tracked
// sweep.  The vertices of a warp lie in one block; every lane of the warp calls
// it.  A template flag, not a test of ref: the 4-lane sweep of a 64 x 64 sheet is
// short enough for the test alone to cost it 0.25 of its 4.4 us.  Sweeps of a
// list whose heads stand unused track nothing.
struct SweepTrack {
    const float4* ref;
    unsigned* moved;
    const int* meta;
};
// whether the heads of a pair list (its meta words) are in use
__device__ __forceinline__ int heads_in_use(const int* meta) { return meta[3]; }
// on: read before the sweep's loads and needed after them
template <bool TRACK>
__device__ __forceinline__ int track_on(const SweepTrack& t) {
    return TRACK ? heads_in_use(t.meta) : 0;
}
template <bool TRACK>
__device__ __forceinline__ void track_motion(const SweepTrack& t, int on, int v, bool valid, float4 out) {
    if (!TRACK || on == 0) return;
    unsigned d2 = 0u;
    if (valid) {
        const float4 ref = __ldg(t.ref + v);
        const float dx = out.x - ref.x, dy = out.y - ref.y, dz = out.z - ref.z;
        d2 = __float_as_uint((dx * dx + dy * dy) + dz * dz);  // a NaN is the largest
    }
    const unsigned m = __reduce_max_sync(0xffffffffu, d2);
    if ((threadIdx.x & 31) == 0 && m != 0u) atomicMax(t.moved + (v >> 5), m);
}

}  // namespace sx
