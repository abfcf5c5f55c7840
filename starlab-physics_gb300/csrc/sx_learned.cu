// Learned warm start for the Jacobi solve (no counterpart in the reference,
// whose substep starts every solve from the predicted positions y,
// XPBD.py:116-118).  A per-vertex MLP 24 -> 64 -> 64 -> 3 (SiLU) maps local
// features of the predicted state to a position correction in units of the
// vertex's mean spring rest length; the solve then starts from
// y + fixed * L * correction.
//
//   features : sx_warm_features     (vertex gather, FP32, stored as BF16[V][32])
//   inference: sx_mlp_forward       (BF16 tensor-core mma, FP32 accumulate,
//                                    activations kept in registers)
//   training : sx_mlp_train_step    (forward + backward data path per 16-row
//                                    tile, weight gradients as dZ^T H products
//                                    on tensor cores, deterministic reduction,
//                                    Adam on FP32 master weights)
//
// Parameter blob (FP32 master, 6792 floats): W1[64][32] | b1[64] | W2[64][64]
// | b2[64] | W3[8][64] | b3[8]; W1's columns 24..31 and W3's rows 3..7 are
// zero.  The BF16 copy holds W1 | W2 | W3 in the same layout.
#include <cuda_bf16.h>

#include "sx_common.cuh"
#include "sx_exact.cuh"

namespace sx {

constexpr int kFeat = 32;   // 24 features + 8 zero columns
constexpr int kHid = 64;
constexpr int kOut = 8;     // 3 used
constexpr int oW1 = 0, ob1 = oW1 + kHid * kFeat, oW2 = ob1 + kHid, ob2 = oW2 + kHid * kHid, oW3 = ob2 + kHid,
              ob3 = oW3 + kOut * kHid, kParams = ob3 + kOut;
constexpr int kW16 = kHid * kFeat + kHid * kHid + kOut * kHid;  // BF16 weights
constexpr int qW1 = 0, qW2 = kHid * kFeat, qW3 = qW2 + kHid * kHid;

__device__ __forceinline__ unsigned short f2bf(float f) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ float bf2f(unsigned short u) { return __bfloat162float(__ushort_as_bfloat16(u)); }
// one packed conversion: the scalar ones run on the special-function unit
__device__ __forceinline__ unsigned pack_bf2(float lo, float hi) {
    unsigned d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// D += A(16x16, row) * B(16x8, col), BF16 inputs, FP32 accumulate.
__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm_x4_trans(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// SiLU, z / (1 + exp(-z)), of a pre-activation, in whose place it leaves the
// derivative s + z s (1 - s), s = 1 / (1 + exp(-z)), from the same reciprocal.  Both
// are correctly rounded quotients (straight-line, sx_exact.cuh: the divisor is at
// least 1, and down to z = -87 below 2^126, where its reciprocal is a normal number);
// below that the reciprocal is 0.  The two minima replace a residual that isn't a
// number, for a divisor and a dividend of infinity: s = 0 and infinity, as the
// divisions give.  (Training step of 65 536 rows 28.1 -> 27.5 us against a quotient of
// its own for the derivative and the exponent capped by one minimum, which let large
// negative values grow without bound; inference by mma, 10^6 rows, 100 -> 103.)
__device__ __forceinline__ float silu(float& z) {
    const float d = 1.0f + expf(-z);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    const float s = __fmaf_rn(y, fminf(__fmaf_rn(-d, y, 1.0f), 1.0f), y);
    const float q = z * s;
    const float r = fminf(__fmaf_rn(-d, q, z), 3.40282347e38f);
    z = s + z * (s * (1.0f - s));
    return __fmaf_rn(r, s, q);
}

// ---------------------------------------------------------------------------
// Features (24, then 8 zeros), from the predicted positions y4, the start of
// substep positions x4, the previous substep's solve correction c4 and the
// constraint adjacency.  L = mean spring rest length at the vertex (Lref).
//   0-2  -(mean over springs of C n) / L        3-5  same over bending pairs
//   6    mean |C|/l0 springs   7 max C/l0   8 min C/l0   9 mean |C|/l0 bending
//   10-12 (y - x)/L            13-15 c/L    16 fixed   17 springs/6  18 bends/6
//   19   |c|/L                 20 |y - x|/L             21-23 g dt^2 / L
// each clamped to [-16, 16] and rounded to BF16.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) warm_features_kernel(int V, const float4* __restrict__ x4,
                                                            const float4* __restrict__ y4,
                                                            const float4* __restrict__ c4,
                                                            const float* __restrict__ fixed,
                                                            const int* __restrict__ ptr,
                                                            const int2* __restrict__ adj,
                                                            const float* __restrict__ Lref, float gx, float gy,
                                                            float gz, float dt, unsigned short* __restrict__ feat,
                                                            float4* __restrict__ ypred) {
    pdl_entry();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const float4 ps = y4[v], xs = x4[v], cp = c4[v];
    if (ypred) ypred[v] = ps;
    const float inv = 1.0f / Lref[v];
    float sx = 0.0f, sy = 0.0f, sz = 0.0f, bx = 0.0f, by = 0.0f, bz = 0.0f;
    float sa = 0.0f, ba = 0.0f, smax = 0.0f, smin = 0.0f;
    int ns = 0, nb = 0;
    const int e = ptr[v + 1];
    for (int k = ptr[v]; k < e; ++k) {
        const int2 a = adj[k];
        const float4 o = y4[a.x & 0x7fffffff];
        const float rest = __int_as_float(a.y);
        const float ex = ps.x - o.x, ey = ps.y - o.y, ez = ps.z - o.z;
        const float l = sqrtf((ex * ex + ey * ey) + ez * ez);
        const float C = l - rest;
        const float il = l > 0.0f ? 1.0f / l : 0.0f;
        const float cx = C * (il * ex), cy = C * (il * ey), cz = C * (il * ez);
        const float r = rest > 0.0f ? C / rest : 0.0f;
        if (a.x < 0) {
            bx = bx + cx; by = by + cy; bz = bz + cz;
            ba = ba + fabsf(r);
            ++nb;
        } else {
            sx = sx + cx; sy = sy + cy; sz = sz + cz;
            sa = sa + fabsf(r);
            smax = ns ? fmaxf(smax, r) : r;
            smin = ns ? fminf(smin, r) : r;
            ++ns;
        }
    }
    const float fs = (float)ns, fb = (float)nb;
    float f[24];
    f[0] = ns ? -((sx / fs) * inv) : 0.0f;
    f[1] = ns ? -((sy / fs) * inv) : 0.0f;
    f[2] = ns ? -((sz / fs) * inv) : 0.0f;
    f[3] = nb ? -((bx / fb) * inv) : 0.0f;
    f[4] = nb ? -((by / fb) * inv) : 0.0f;
    f[5] = nb ? -((bz / fb) * inv) : 0.0f;
    f[6] = ns ? sa / fs : 0.0f;
    f[7] = smax;
    f[8] = smin;
    f[9] = nb ? ba / fb : 0.0f;
    const float dx = ps.x - xs.x, dy = ps.y - xs.y, dz = ps.z - xs.z;
    f[10] = dx * inv;
    f[11] = dy * inv;
    f[12] = dz * inv;
    f[13] = cp.x * inv;
    f[14] = cp.y * inv;
    f[15] = cp.z * inv;
    f[16] = fixed[v];
    f[17] = fs / 6.0f;
    f[18] = fb / 6.0f;
    f[19] = sqrtf((cp.x * cp.x + cp.y * cp.y) + cp.z * cp.z) * inv;
    f[20] = sqrtf((dx * dx + dy * dy) + dz * dz) * inv;
    f[21] = ((gx * dt) * dt) * inv;
    f[22] = ((gy * dt) * dt) * inv;
    f[23] = ((gz * dt) * dt) * inv;
    unsigned* out = reinterpret_cast<unsigned*>(feat + (size_t)v * kFeat);
#pragma unroll
    for (int i = 0; i < 12; ++i)
        out[i] = pack_bf2(fminf(fmaxf(f[2 * i], -16.0f), 16.0f), fminf(fmaxf(f[2 * i + 1], -16.0f), 16.0f));
#pragma unroll
    for (int i = 12; i < 16; ++i) out[i] = 0u;
}

// y = y_pred + fixed * (L * d) for the first three outputs d of the MLP.
__global__ void warm_apply_kernel(int V, const float4* __restrict__ ypred, const float* __restrict__ out4,
                                  const float* __restrict__ fixed, const float* __restrict__ Lref,
                                  float4* __restrict__ y4) {
    pdl_entry();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const float4 p = ypred[v];
    const float f = fixed[v], L = Lref[v];
    float4 y = p;
    y.x = p.x + f * (L * out4[4 * v]);
    y.y = p.y + f * (L * out4[4 * v + 1]);
    y.z = p.z + f * (L * out4[4 * v + 2]);
    y4[v] = y;
}

// After the solve: c = y - y_pred (the next substep's feature 13-15) and the
// training target (c / L, fixed) as float4.
__global__ void warm_record_kernel(int V, const float4* __restrict__ y4, const float4* __restrict__ ypred,
                                   const float* __restrict__ fixed, const float* __restrict__ Lref,
                                   float4* __restrict__ c4, float4* __restrict__ target4) {
    pdl_entry();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const float4 y = y4[v], p = ypred[v];
    const float4 c = make_float4(y.x - p.x, y.y - p.y, y.z - p.z, 0.0f);
    c4[v] = c;
    if (target4) {
        const float inv = 1.0f / Lref[v];
        target4[v] = make_float4(c.x * inv, c.y * inv, c.z * inv, fixed[v]);
    }
}

// If the warm start raised the residual (res_warm[2] > res_cold[2]), restore
// the cold start y = y_pred; flag[0] counts fallbacks, flag[1] warm starts.
__global__ void warm_select_kernel(int V, const double* __restrict__ res_warm, const double* __restrict__ res_cold,
                                   const float4* __restrict__ ypred, float4* __restrict__ y4, int* flag) {
    pdl_entry();
    const bool cold = res_warm[2] > res_cold[2];
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v == 0) {
        if (cold) flag[0] += 1;
        else flag[1] += 1;
    }
    if (cold && v < V) y4[v] = ypred[v];
}

// ---------------------------------------------------------------------------
// MLP tiles.  A warp owns 16 rows.  Shared weights (BF16, rows padded so that
// the fragment loads are bank-conflict free):
//   W1s[64][40] (n, k), W2s[64][72] (n, k), W3s[8][72] (n, k);
// the backward data path reads W2 and W3 transposed by ldmatrix.trans.
// ---------------------------------------------------------------------------
constexpr int S1 = 40, S2 = 72, S3 = 72;

struct MlpSmem {
    alignas(16) unsigned short W1[kHid * S1];
    alignas(16) unsigned short W2[kHid * S2];
    alignas(16) unsigned short W3[kOut * S3];
    float b1[kHid], b2[kHid], b3[kOut];
};
// rows of K values to rows of the padded stride, 16 bytes at a time where the
// source allows it
__device__ __forceinline__ void stage_rows(unsigned short* dst, int stride, const unsigned short* __restrict__ src,
                                           int rows, int K, bool wide) {
    if (wide) {
        for (int i = threadIdx.x; i < rows * (K / 8); i += blockDim.x) {
            const int n = i / (K / 8), k = i % (K / 8) * 8;
            *reinterpret_cast<uint4*>(dst + n * stride + k) = *reinterpret_cast<const uint4*>(src + n * K + k);
        }
    } else {
        for (int i = threadIdx.x; i < rows * K; i += blockDim.x) dst[i / K * stride + i % K] = src[i];
    }
}
__device__ void stage_weights(MlpSmem& s, const unsigned short* __restrict__ w16, const float* __restrict__ p32) {
    const bool wide = (reinterpret_cast<uintptr_t>(w16) & 15) == 0;
    stage_rows(s.W1, S1, w16 + qW1, kHid, kFeat, wide);
    stage_rows(s.W2, S2, w16 + qW2, kHid, kHid, wide);
    stage_rows(s.W3, S3, w16 + qW3, kOut, kHid, wide);
    for (int i = threadIdx.x; i < kHid; i += blockDim.x) {
        s.b1[i] = p32[ob1 + i];
        s.b2[i] = p32[ob2 + i];
    }
    if (threadIdx.x < kOut) s.b3[threadIdx.x] = p32[ob3 + threadIdx.x];
}

__device__ __forceinline__ unsigned lds32(const unsigned short* p) { return *reinterpret_cast<const unsigned*>(p); }

// Forward of one 16-row tile.  X rows: feature row of tile row r is
// xrow(r) (or -1 for padding rows).  Outputs the derivatives of both layers'
// SiLU at their pre-activations (C layout) and O (C layout, 8 columns).
struct Frag64 {
    float c[8][4];
};

// keep(layer, ks, a): the activations of hidden layer 1 or 2 as A fragments
// (rows g, g + 8 of columns 16 ks + 2 tig, then the same 8 columns on).
template <typename Keep>
__device__ __forceinline__ void tile_forward(const MlpSmem& s, const unsigned (&ax)[2][4], Frag64& z1, Frag64& z2,
                                             float (&o)[4], Keep keep) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float b0 = s.b1[8 * j + 2 * tig], b1v = s.b1[8 * j + 2 * tig + 1];
        z1.c[j][0] = b0; z1.c[j][1] = b1v; z1.c[j][2] = b0; z1.c[j][3] = b1v;
    }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const unsigned short* w = s.W1 + (8 * j + g) * S1 + 16 * ks + 2 * tig;
            mma16816(z1.c[j], ax[ks], lds32(w), lds32(w + 8));
        }
    unsigned ah[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        ah[ks][0] = pack_bf2(silu(z1.c[2 * ks][0]), silu(z1.c[2 * ks][1]));
        ah[ks][1] = pack_bf2(silu(z1.c[2 * ks][2]), silu(z1.c[2 * ks][3]));
        ah[ks][2] = pack_bf2(silu(z1.c[2 * ks + 1][0]), silu(z1.c[2 * ks + 1][1]));
        ah[ks][3] = pack_bf2(silu(z1.c[2 * ks + 1][2]), silu(z1.c[2 * ks + 1][3]));
        keep(1, ks, ah[ks]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float b0 = s.b2[8 * j + 2 * tig], b1v = s.b2[8 * j + 2 * tig + 1];
        z2.c[j][0] = b0; z2.c[j][1] = b1v; z2.c[j][2] = b0; z2.c[j][3] = b1v;
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const unsigned short* w = s.W2 + (8 * j + g) * S2 + 16 * ks + 2 * tig;
            mma16816(z2.c[j], ah[ks], lds32(w), lds32(w + 8));
        }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        ah[ks][0] = pack_bf2(silu(z2.c[2 * ks][0]), silu(z2.c[2 * ks][1]));
        ah[ks][1] = pack_bf2(silu(z2.c[2 * ks][2]), silu(z2.c[2 * ks][3]));
        ah[ks][2] = pack_bf2(silu(z2.c[2 * ks + 1][0]), silu(z2.c[2 * ks + 1][1]));
        ah[ks][3] = pack_bf2(silu(z2.c[2 * ks + 1][2]), silu(z2.c[2 * ks + 1][3]));
        keep(2, ks, ah[ks]);
    }
    o[0] = s.b3[2 * tig]; o[1] = s.b3[2 * tig + 1]; o[2] = o[0]; o[3] = o[1];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const unsigned short* w = s.W3 + g * S3 + 16 * ks + 2 * tig;
        mma16816(o, ah[ks], lds32(w), lds32(w + 8));
    }
}

// A fragments of a 16-row tile of BF16 features (rows r0+g, r0+g+8).
__device__ __forceinline__ void load_x_frag(const unsigned short* __restrict__ feat, int ra, int rb,
                                            unsigned (&ax)[2][4]) {
    const int tig = threadIdx.x & 3;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        const int c = 16 * ks + 2 * tig;
        ax[ks][0] = ra >= 0 ? *reinterpret_cast<const unsigned*>(feat + (size_t)ra * kFeat + c) : 0u;
        ax[ks][1] = rb >= 0 ? *reinterpret_cast<const unsigned*>(feat + (size_t)rb * kFeat + c) : 0u;
        ax[ks][2] = ra >= 0 ? *reinterpret_cast<const unsigned*>(feat + (size_t)ra * kFeat + c + 8) : 0u;
        ax[ks][3] = rb >= 0 ? *reinterpret_cast<const unsigned*>(feat + (size_t)rb * kFeat + c + 8) : 0u;
    }
}

constexpr int MLP_BLOCK = 128;

__global__ void __launch_bounds__(MLP_BLOCK) mlp_forward_kernel(int V, const unsigned short* __restrict__ feat,
                                                                const unsigned short* __restrict__ w16,
                                                                const float* __restrict__ p32,
                                                                float* __restrict__ out4) {
    pdl_entry();
    __shared__ MlpSmem s;
    stage_weights(s, w16, p32);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int r0 = warp * 16; r0 < V; r0 += nwarps * 16) {
        const int ra = r0 + g < V ? r0 + g : -1, rb = r0 + g + 8 < V ? r0 + g + 8 : -1;
        unsigned ax[2][4];
        load_x_frag(feat, ra, rb, ax);
        Frag64 z1, z2;
        float o[4];
        tile_forward(s, ax, z1, z2, o, [](int, int, const unsigned(&)[4]) {});
        if (tig < 2) {
            if (ra >= 0) *reinterpret_cast<float2*>(out4 + 4 * (size_t)ra + 2 * tig) = make_float2(o[0], o[1]);
            if (rb >= 0) *reinterpret_cast<float2*>(out4 + 4 * (size_t)rb + 2 * tig) = make_float2(o[2], o[3]);
        }
    }
}

// ---------------------------------------------------------------------------
// Inference on the 5th-generation tensor cores (tcgen05).  One CTA of 256
// threads takes 128 rows at a time (M = 128; two threads per row, one per
// half of the 64 hidden columns): the rows' features, the hidden
// activations and the three weight matrices sit in shared memory in the
// canonical no-swizzle K-major layout (8 x 16-byte core matrices; LBO = 128 B
// between core matrices along K, SBO = (K / 8) x 128 B between 8-row groups);
// thread 0 issues tcgen05.mma (kind::f16, BF16 x BF16 -> FP32) into tensor
// memory, whose completion tcgen05.commit signals on an mbarrier; each warp
// then reads its 32 rows of the accumulator with tcgen05.ld, adds the bias,
// applies SiLU, and writes the next layer's BF16 operand over the last one.
// Layer 3 is N = 16 (W3's 8 rows and 8 zero rows); one accumulator of 64
// tensor-memory columns per CTA serves all three layers, each read before the
// next overwrites it.
//
// The special-function unit sets the floor: 128 tanh a row, 16 a clock and SM, 26
// us for 10^6 rows.  So nothing else may run on it (the scalar float to BF16
// conversion does; the packed one does not: 77 -> 53 us), and the CTAs of an SM
// have to keep it fed through each other's waits: one block barrier per layer,
// the next tile's features loaded a tile ahead, packed two-wide float operations,
// and waits on the mbarrier's own suspended try_wait.  10^6 rows take 52 us, 8 of
// them before the first tile's end (97 with two block barriers per layer, a
// global timer read in every thread's wait, no prefetch and scalar conversions).
// 4, 5 or 6 CTAs per SM give 53, 52 and 54 us; ex2 and half a reciprocal in the
// place of tanh 59; plain loads of a row by its own two threads are faster than
// coalesced ones regrouped in shared memory (52 against 55).
//
// Every wait is bounded (TC_TRIES tries, each suspended for up to 10 us); one that
// gives up sets SX_STATUS_WAIT_TIMEOUT, waits once more (bounded) for the MMAs
// in flight, frees the tensor memory and ends the kernel.
// ---------------------------------------------------------------------------
constexpr int TC_ROWS = 128;
constexpr int TC_THREADS = 256;  // warp w reads tensor-memory lanes 32 (w % 4).., columns half w / 4
constexpr int TC_TMEM_COLS = 64;   // every layer's accumulator: the last one has been read by then
constexpr int TC_PER_SM = 5;       // CTAs: 48 registers a thread, 31 KB of shared memory

struct TcSmem {
    alignas(128) unsigned short A[TC_ROWS * kHid];  // features, then hidden activations
    alignas(128) unsigned short B1[kHid * kFeat];
    alignas(128) unsigned short B2[kHid * kHid];
    alignas(128) unsigned short B3[16 * kHid];
    alignas(16) float b1[kHid], b2[kHid];
    float b3[16];
    alignas(8) unsigned long long bar;
    unsigned tmem_base;
};

// element (r, k) of a K-major operand with K columns, canonical layout
__device__ __forceinline__ int canon(int r, int k, int K) {
    return ((r >> 3) * (K >> 3) + (k >> 3)) * 64 + (r & 7) * 8 + (k & 7);
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// shared-memory matrix descriptor: start, LBO, SBO (16-byte units), version 1, no swizzle
__device__ __forceinline__ unsigned long long umma_sdesc(unsigned saddr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((saddr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
           ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor, kind::f16: D F32, A and B BF16, both K-major
__host__ __device__ constexpr unsigned umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(N >> 3) << 17) | ((unsigned)(M >> 4) << 24);
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void umma_bf16(unsigned d_tmem, unsigned long long a, unsigned long long b, unsigned idesc,
                                          unsigned accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
constexpr int TC_TRIES = 1 << 18;
// a try suspends the thread until the phase completes or the hint (ns) is over
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(10000u)
        : "memory");
    return done != 0u;
}
__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity) {
    for (int k = 0; k < TC_TRIES; ++k)
        if (mbar_try(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld4(unsigned taddr, unsigned (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Packed float pairs: the same rounding as two scalar operations.
#define SX_F32X2(name, op)                                                                                    \
    __device__ __forceinline__ float2 name(float2 a, float2 b) {                                              \
        float2 d;                                                                                             \
        asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t" op                \
            " w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}"                                                         \
            : "=f"(d.x), "=f"(d.y)                                                                            \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                        \
        return d;                                                                                             \
    }
SX_F32X2(add2, "add.rn.f32x2")
SX_F32X2(mul2, "mul.rn.f32x2")
#undef SX_F32X2
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
// SiLU through the hardware tanh: z * sigmoid(z) = h + h * tanh(h) with
// h = z / 2, one special-function instruction instead of an exponential and a
// reciprocal.  The tensor-core path's hidden activations are rounded to BF16, far
// coarser than tanh.approx's error.
__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 silu2(float2 z) {
    const float2 h = mul2(z, make_float2(0.5f, 0.5f));
    return fma2(h, make_float2(tanh_hw(h.x), tanh_hw(h.y)), h);
}

// 32 accumulator columns of this thread's row (at taddr) + bias -> SiLU ->
// BF16 columns [c0, c0 + 32) of row `row` of A; 16 at a time, which keeps the
// kernel at 48 registers
__device__ __forceinline__ void tc_hidden_half(unsigned taddr, const float* bias, unsigned short* A, int row, int c0) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        unsigned r[16];
        tmem_ld16(taddr + 16 * p, r);
        const float2* b2 = reinterpret_cast<const float2*>(bias + c0 + 16 * p);
        tmem_wait_ld();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint4 v;
            unsigned* pv = reinterpret_cast<unsigned*>(&v);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = 8 * q + 2 * e;
                const float2 y = silu2(add2(make_float2(__uint_as_float(r[c]), __uint_as_float(r[c + 1])), b2[c / 2]));
                pv[e] = pack_bf2(y.x, y.y);
            }
            *reinterpret_cast<uint4*>(A + canon(row, c0 + 16 * p + 8 * q, kHid)) = v;
        }
    }
}

// 8 consecutive k of row n of a weight matrix -> its 16 bytes of the canonical layout
__device__ __forceinline__ void stage_canon(unsigned short* dst, const unsigned short* __restrict__ src, int rows,
                                            int zero_from, int K, bool wide) {
    for (int i = threadIdx.x; i < rows * (K / 8); i += TC_THREADS) {
        const int n = i / (K / 8), k = i % (K / 8) * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (n < zero_from) {
            if (wide) {
                v = *reinterpret_cast<const uint4*>(src + n * K + k);
            } else {
                unsigned short* h = reinterpret_cast<unsigned short*>(&v);
#pragma unroll
                for (int j = 0; j < 8; ++j) h[j] = src[n * K + k + j];
            }
        }
        *reinterpret_cast<uint4*>(dst + canon(n, k, K)) = v;
    }
}

__global__ void __launch_bounds__(TC_THREADS, TC_PER_SM) mlp_forward_tc_kernel(int V, const unsigned short* __restrict__ feat,
                                                                    const unsigned short* __restrict__ w16,
                                                                    const float* __restrict__ p32,
                                                                    float* __restrict__ out4, int* status) {
    pdl_entry();
    __shared__ TcSmem s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = warp & 3, half = warp >> 2;
    const int trow = 32 * quad + lane;  // this thread's row within a tile
    const bool wide = (reinterpret_cast<uintptr_t>(w16) & 15) == 0;
    stage_canon(s.B1, w16 + qW1, kHid, kHid, kFeat, wide);
    stage_canon(s.B2, w16 + qW2, kHid, kHid, kHid, wide);
    stage_canon(s.B3, w16 + qW3, 16, kOut, kHid, wide);
    for (int i = tid; i < kHid; i += TC_THREADS) {
        s.b1[i] = p32[ob1 + i];
        s.b2[i] = p32[ob2 + i];
    }
    if (tid < 16) s.b3[tid] = tid < kOut ? p32[ob3 + tid] : 0.0f;
    const unsigned bar = smem_u32(&s.bar);
    if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tbase = s.tmem_base;
    const unsigned lane_row = (unsigned)(32 * quad) << 16;  // this warp's 32 tensor-memory lanes
    const unsigned long long dB1 = umma_sdesc(smem_u32(s.B1), 128, 512);
    const unsigned long long dB2 = umma_sdesc(smem_u32(s.B2), 128, 1024);
    const unsigned long long dB3 = umma_sdesc(smem_u32(s.B3), 128, 1024);
    const unsigned long long dA1 = umma_sdesc(smem_u32(s.A), 128, 512);
    const unsigned long long dA2 = umma_sdesc(smem_u32(s.A), 128, 1024);
    constexpr unsigned id64 = umma_idesc_bf16(TC_ROWS, kHid), id16 = umma_idesc_bf16(TC_ROWS, 16);
    unsigned phase = 0;
    bool ok = true;
    const long long ntiles = ((long long)V + TC_ROWS - 1) / TC_ROWS;
    // half a row of features (16 BF16) per thread
    uint4 f[2];
    auto load_features = [&](long long tile) {
        const long long row = tile * TC_ROWS + trow;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            f[j] = tile < ntiles && row < V
                       ? __ldg(reinterpret_cast<const uint4*>(feat + (size_t)row * kFeat) + 2 * half + j)
                       : make_uint4(0, 0, 0, 0);
    };
    // this thread's shared-memory stores and tensor-memory loads are done: one
    // barrier, and thread 0 issues the next layer; false when a wait gave up
    auto publish = [&]() {
        fence_async_smem();
        tc_fence_before();
        return __syncthreads_and(ok) != 0;
    };
    load_features(blockIdx.x);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
#pragma unroll
        for (int j = 0; j < 2; ++j) *reinterpret_cast<uint4*>(s.A + canon(trow, 16 * half + 8 * j, kFeat)) = f[j];
        // (the last tile's layer-3 accumulator, where D1 goes, has been read
        // before this barrier)
        if (!publish()) break;
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < kFeat / 16; ++ks) umma_bf16(tbase, dA1 + 16 * ks, dB1 + 16 * ks, id64, ks);
            umma_commit(bar);
        }
        load_features(tile + gridDim.x);
        ok = mbar_wait_bounded(bar, phase);
        phase ^= 1u;
        tc_fence_after();
        tc_hidden_half(tbase + lane_row + 32 * half, s.b1, s.A, trow, 32 * half);
        if (!publish()) break;
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < kHid / 16; ++ks) umma_bf16(tbase, dA2 + 16 * ks, dB2 + 16 * ks, id64, ks);
            umma_commit(bar);
        }
        ok = mbar_wait_bounded(bar, phase);
        phase ^= 1u;
        tc_fence_after();
        tc_hidden_half(tbase + lane_row + 32 * half, s.b2, s.A, trow, 32 * half);  // layer 2 is done with A2
        if (!publish()) break;
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < kHid / 16; ++ks) umma_bf16(tbase, dA2 + 16 * ks, dB3 + 16 * ks, id16, ks);
            umma_commit(bar);
        }
        ok = mbar_wait_bounded(bar, phase);
        phase ^= 1u;
        tc_fence_after();
        if (half == 0) {
            unsigned r[4];
            tmem_ld4(tbase + lane_row, r);
            tmem_wait_ld();
            const long long row = tile * TC_ROWS + trow;
            if (row < V)
                *reinterpret_cast<float4*>(out4 + 4 * (size_t)row) =
                    make_float4(__uint_as_float(r[0]) + s.b3[0], __uint_as_float(r[1]) + s.b3[1],
                                __uint_as_float(r[2]) + s.b3[2], __uint_as_float(r[3]) + s.b3[3]);
        }
    }
    // a wait that gave up: the last layer's MMAs may be in flight, once more
    // within the bound
    ok = __syncthreads_and(ok) != 0;
    if (!ok) {
        if (tid == 0) atomicOr(status, SX_STATUS_WAIT_TIMEOUT);
        mbar_wait_bounded(bar, phase ^ 1u);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TC_TMEM_COLS)
                     : "memory");
}

// ---------------------------------------------------------------------------
// Training, part 1: forward, backward and weight gradients of a minibatch.  Rows
// are idx[i] into the sample arrays (feat, target4 = (t, mask)).  Loss = sum over
// rows and the 3 outputs of mask * (o - t)^2 / n_valid.
//
// A block takes tiles of 64 rows, a warp 16 of them: forward and backward data
// path on its own rows with activations in registers, everything the weight
// gradients need (X, H1, H2, dZ1, dZ2, dO, BF16) to shared memory; then dW1 =
// dZ1^T X, dW2 = dZ2^T H1 and dW3 = dO^T H2 over the tile (A and B fragments by
// ldmatrix.trans), warp w owning output rows 16 w .. of dW1 and dW2 and columns 16
// w .. of dW3, accumulated in registers over the block's tiles.  One partial of
// all parameters and the loss per block.
//
// The rows are few (65 536 are 1 024 tiles, 3.4 per block), so latency bounds it:
// weights are staged 16 bytes at a time and only once, the next tile's features
// load a tile ahead, and nothing returns to global memory in between.  (As two
// kernels, with transposed weight copies staged value by value, activations and
// gradients through global memory and bias partials per warp: 66 + 40 us, and 23
// for the reduction over 4 096 warps' partials.)
// ---------------------------------------------------------------------------
constexpr int TR_ROWS = 64, TR_PER_SM = 2;
constexpr int SL = 72, SX = 40, SD = 24;  // padded row strides (BF16) of 64, 32 and 16 columns
constexpr int kBias = 1 + kHid + kHid + kOut;  // loss, db1, db2, db3
constexpr int kPart = kParams + 1;             // a block's partial: the parameters in order, then the loss

struct TrainSmem {
    MlpSmem w;
    alignas(16) unsigned short X[TR_ROWS * SX];
    alignas(16) unsigned short H1[TR_ROWS * SL], H2[TR_ROWS * SL], D1[TR_ROWS * SL], D2[TR_ROWS * SL];
    alignas(16) unsigned short DO[TR_ROWS * SD];  // columns 8 .. 15 zero
    float bias[MLP_BLOCK / 32][kBias];
};

// sum over the 8 row groups g of a C-fragment column pair (lanes with equal tig)
__device__ __forceinline__ float colsum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

__global__ void __launch_bounds__(MLP_BLOCK, TR_PER_SM) mlp_train_kernel(int M, const int* __restrict__ idx,
                                                                         const unsigned short* __restrict__ feat,
                                                                         const float4* __restrict__ target4,
                                                                         float inv_valid,
                                                                         const unsigned short* __restrict__ w16,
                                                                         const float* __restrict__ p32,
                                                                         float* __restrict__ part) {
    pdl_entry();
    extern __shared__ uint4 smem_raw[];
    TrainSmem& s = *reinterpret_cast<TrainSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, tig = lane & 3;
    const int q = lane >> 3, r8 = lane & 7;
    // the warp's 16 feature rows of a tile: 64 pieces of 16 bytes, two a lane
    auto piece = [&](int j) { return lane + 32 * j; };
    auto load_idx = [&](long long tile, int (&id)[2]) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const long long row = tile * TR_ROWS + 16 * w + (piece(j) >> 2);
            id[j] = row < M ? idx[row] : -1;
        }
    };
    auto load_x = [&](const int (&id)[2], uint4 (&x)[2]) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
            x[j] = id[j] >= 0 ? *reinterpret_cast<const uint4*>(feat + (size_t)id[j] * kFeat + (piece(j) & 3) * 8)
                              : make_uint4(0u, 0u, 0u, 0u);
    };
    const long long ntiles = ((long long)M + TR_ROWS - 1) / TR_ROWS;
    int id[2], next[2];
    uint4 x[2];
    load_idx(blockIdx.x, id);
    load_idx(blockIdx.x + gridDim.x, next);
    stage_weights(s.w, w16, p32);
    for (int i = threadIdx.x; i < TR_ROWS; i += MLP_BLOCK)
        *reinterpret_cast<uint4*>(s.DO + i * SD + 8) = make_uint4(0u, 0u, 0u, 0u);
    load_x(id, x);
    __syncthreads();

    float a1[4][4], a2[8][4], a3[2][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) a2[j][0] = a2[j][1] = a2[j][2] = a2[j][3] = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) a1[j][0] = a1[j][1] = a1[j][2] = a1[j][3] = 0.0f;
#pragma unroll
    for (int j = 0; j < 2; ++j) a3[j][0] = a3[j][1] = a3[j][2] = a3[j][3] = 0.0f;
    float loss = 0.0f, db1[8][2], db2[8][2], db3[2];
#pragma unroll
    for (int j = 0; j < 8; ++j) db1[j][0] = db1[j][1] = db2[j][0] = db2[j][1] = 0.0f;
    db3[0] = db3[1] = 0.0f;
    const int ra = 16 * w + g, rb = ra + 8;  // this lane's rows of the tile
    auto put = [](unsigned short* p, unsigned v) { *reinterpret_cast<unsigned*>(p) = v; };

    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int sa = __shfl_sync(0xffffffffu, id[0], 4 * g), sb = __shfl_sync(0xffffffffu, id[1], 4 * g);
        float4 ta = make_float4(0.f, 0.f, 0.f, 0.f), tb = ta;
        if (tig < 2) {
            if (sa >= 0) ta = target4[sa];
            if (sb >= 0) tb = target4[sb];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
            *reinterpret_cast<uint4*>(s.X + (16 * w + (piece(j) >> 2)) * SX + (piece(j) & 3) * 8) = x[j];
        __syncwarp();
        id[0] = next[0];
        id[1] = next[1];
        load_x(id, x);
        load_idx(tile + 2LL * gridDim.x, next);
        unsigned ax[2][4];
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const int c = 16 * ks + 2 * tig;
            ax[ks][0] = lds32(s.X + ra * SX + c);
            ax[ks][1] = lds32(s.X + rb * SX + c);
            ax[ks][2] = lds32(s.X + ra * SX + c + 8);
            ax[ks][3] = lds32(s.X + rb * SX + c + 8);
        }
        Frag64 z1, z2;
        float o[4];
        tile_forward(s.w, ax, z1, z2, o, [&](int layer, int ks, const unsigned(&a)[4]) {
            unsigned short* h = layer == 1 ? s.H1 : s.H2;
            const int c = 16 * ks + 2 * tig;
            put(h + ra * SL + c, a[0]);
            put(h + rb * SL + c, a[1]);
            put(h + ra * SL + c + 8, a[2]);
            put(h + rb * SL + c + 8, a[3]);
        });
        // dO (C layout: rows g, g+8; columns 2tig, 2tig+1)
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (tig < 2) {
            const float tta[4] = {ta.x, ta.y, ta.z, 0.0f}, ttb[4] = {tb.x, tb.y, tb.z, 0.0f};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int col = 2 * tig + u;
                if (col < 3) {
                    const float ea = ta.w * (o[u] - tta[col]), eb = tb.w * (o[2 + u] - ttb[col]);
                    loss = loss + (ea * (o[u] - tta[col]) + eb * (o[2 + u] - ttb[col]));
                    d[u] = (2.0f * inv_valid) * ea;
                    d[2 + u] = (2.0f * inv_valid) * eb;
                }
            }
        }
        db3[0] += d[0] + d[2];
        db3[1] += d[1] + d[3];
        // dH2 = dO W3 (K = 16, columns 8..15 of dO are zero), dZ2 = dH2 * silu'(Z2)
        const unsigned ad[4] = {pack_bf2(d[0], d[1]), pack_bf2(d[2], d[3]), 0u, 0u};
        put(s.DO + ra * SD + 2 * tig, ad[0]);
        put(s.DO + rb * SD + 2 * tig, ad[1]);
        unsigned az[4][4];
#pragma unroll
        for (int jq = 0; jq < 2; ++jq) {
            unsigned B[4];  // W3 rows 0..7 (k), columns 8 j .. of j = 4 jq .. 4 jq + 3
            ldsm_x4_trans(B, s.w.W3 + r8 * S3 + 8 * (4 * jq + q));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = 4 * jq + i;
                float dz[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma16816(dz, ad, B[i], 0u);
#pragma unroll
                for (int u = 0; u < 4; ++u) dz[u] = dz[u] * z2.c[j][u];
                db2[j][0] += dz[0] + dz[2];
                db2[j][1] += dz[1] + dz[3];
                const unsigned lo = pack_bf2(dz[0], dz[1]), hi = pack_bf2(dz[2], dz[3]);
                az[j / 2][2 * (j & 1)] = lo;
                az[j / 2][2 * (j & 1) + 1] = hi;
                put(s.D2 + ra * SL + 8 * j + 2 * tig, lo);
                put(s.D2 + rb * SL + 8 * j + 2 * tig, hi);
            }
        }
        // dH1 = dZ2 W2, dZ1 = dH1 * silu'(Z1)
#pragma unroll
        for (int jp = 0; jp < 4; ++jp) {
            float c[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                unsigned B[4];  // W2 rows 16 ks .. (k), columns 16 jp ..: (k, n) (k+8, n) (k, n+8) (k+8, n+8)
                ldsm_x4_trans(B, s.w.W2 + (16 * ks + (q & 1) * 8 + r8) * S2 + 16 * jp + (q >> 1) * 8);
                mma16816(c[0], az[ks], B[0], B[1]);
                mma16816(c[1], az[ks], B[2], B[3]);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int j = 2 * jp + i;
#pragma unroll
                for (int u = 0; u < 4; ++u) c[i][u] = c[i][u] * z1.c[j][u];
                db1[j][0] += c[i][0] + c[i][2];
                db1[j][1] += c[i][1] + c[i][3];
                put(s.D1 + ra * SL + 8 * j + 2 * tig, pack_bf2(c[i][0], c[i][1]));
                put(s.D1 + rb * SL + 8 * j + 2 * tig, pack_bf2(c[i][2], c[i][3]));
            }
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < TR_ROWS / 16; ++ks) {
            const int m0 = 16 * ks;
            // A = D^T rows o0 = 16w .. 16w+15 (matrices: (m0,o0) (m0,o0+8) (m0+8,o0) (m0+8,o0+8))
            const int am = m0 + (q >> 1) * 8 + r8, ao = 16 * w + (q & 1) * 8;
            unsigned A2[4], A1[4];
            ldsm_x4_trans(A2, s.D2 + am * SL + ao);
            ldsm_x4_trans(A1, s.D1 + am * SL + ao);
            // B fragments for two n-tiles per load: matrices (m0,n0) (m0+8,n0) (m0,n0+8) (m0+8,n0+8)
            const int bm = m0 + (q & 1) * 8 + r8, bn = (q >> 1) * 8;
#pragma unroll
            for (int jp = 0; jp < 4; ++jp) {
                unsigned B[4];
                ldsm_x4_trans(B, s.H1 + bm * SL + 16 * jp + bn);
                mma16816(a2[2 * jp], A2, B[0], B[1]);
                mma16816(a2[2 * jp + 1], A2, B[2], B[3]);
            }
#pragma unroll
            for (int jp = 0; jp < 2; ++jp) {
                unsigned B[4];
                ldsm_x4_trans(B, s.X + bm * SX + 16 * jp + bn);
                mma16816(a1[2 * jp], A1, B[0], B[1]);
                mma16816(a1[2 * jp + 1], A1, B[2], B[3]);
            }
            // dW3: A = dO^T (16 rows, 8 used), B = H2 columns 16w .. 16w+15
            unsigned A3[4], B3[4];
            ldsm_x4_trans(A3, s.DO + am * SD + (q & 1) * 8);
            ldsm_x4_trans(B3, s.H2 + bm * SL + 16 * w + bn);
            mma16816(a3[0], A3, B3[0], B3[1]);
            mma16816(a3[1], A3, B3[2], B3[3]);
        }
        __syncthreads();
    }
    // bias gradients and loss: over the lanes, then over the warps in order
    float* wb = s.bias[w];
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
    if (lane == 0) wb[0] = loss;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float u0 = colsum(db1[j][0]), u1 = colsum(db1[j][1]);
        const float v0 = colsum(db2[j][0]), v1 = colsum(db2[j][1]);
        if (g == 0) {
            wb[1 + 8 * j + 2 * tig] = u0;
            wb[1 + 8 * j + 2 * tig + 1] = u1;
            wb[1 + kHid + 8 * j + 2 * tig] = v0;
            wb[1 + kHid + 8 * j + 2 * tig + 1] = v1;
        }
    }
    const float e0 = colsum(db3[0]), e1 = colsum(db3[1]);
    if (g == 0) {
        wb[1 + 2 * kHid + 2 * tig] = e0;
        wb[1 + 2 * kHid + 2 * tig + 1] = e1;
    }
    __syncthreads();
    float* bp = part + (size_t)blockIdx.x * kPart;
    for (int i = threadIdx.x; i < kBias; i += MLP_BLOCK) {
        float t = s.bias[0][i];
#pragma unroll
        for (int k = 1; k < MLP_BLOCK / 32; ++k) t += s.bias[k][i];
        const int at = i == 0            ? kParams
                       : i < 1 + kHid     ? ob1 + i - 1
                       : i < 1 + 2 * kHid ? ob2 + i - 1 - kHid
                                          : ob3 + i - 1 - 2 * kHid;
        bp[at] = t;
    }
    // weight gradients (C layout: rows g, g+8; columns 2tig, 2tig+1)
    const int o_lo = 16 * w + g, o_hi = o_lo + 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = 8 * j + 2 * tig;
        bp[oW1 + o_lo * kFeat + c] = a1[j][0];
        bp[oW1 + o_lo * kFeat + c + 1] = a1[j][1];
        bp[oW1 + o_hi * kFeat + c] = a1[j][2];
        bp[oW1 + o_hi * kFeat + c + 1] = a1[j][3];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = 8 * j + 2 * tig;
        bp[oW2 + o_lo * kHid + c] = a2[j][0];
        bp[oW2 + o_lo * kHid + c + 1] = a2[j][1];
        bp[oW2 + o_hi * kHid + c] = a2[j][2];
        bp[oW2 + o_hi * kHid + c + 1] = a2[j][3];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int c = 16 * w + 8 * j + 2 * tig;
        if (g < kOut) {
            bp[oW3 + g * kHid + c] = a3[j][0];
            bp[oW3 + g * kHid + c + 1] = a3[j][1];
        }
    }
}

// ---------------------------------------------------------------------------
// Training, part 2: sum the blocks' partials in a fixed order into grad;
// stats[0] = loss.
// Part 3: Adam on the FP32 master weights, refreshing the BF16 copy.
// Structurally zero parameters (W1 columns >= 24, W3/b3 rows >= 3) stay zero.
// ---------------------------------------------------------------------------
constexpr int RD_GROUPS = 16;  // partial groups per parameter column in mlp_reduce_kernel

// Block = 32 parameter columns x RD_GROUPS groups: group y sums partials
// y, y + RD_GROUPS, ... of its column (coalesced across the columns), then
// the groups are added in order -- a fixed order, so the sums are
// deterministic.
__global__ void __launch_bounds__(32 * RD_GROUPS) mlp_reduce_kernel(int nblocks, const float* __restrict__ part,
                                                                   float* __restrict__ grad,
                                                                   float* __restrict__ stats) {
    pdl_entry();
    __shared__ float sums[RD_GROUPS][33];
    const int tx = threadIdx.x & 31, gy = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + tx;
    float sum = 0.0f;
    if (i < kPart) {
#pragma unroll 8
        for (int k = gy; k < nblocks; k += RD_GROUPS) sum += part[(size_t)k * kPart + i];
    }
    sums[gy][tx] = sum;
    __syncthreads();
    if (gy == 0 && i < kPart) {
        float t = sums[0][tx];
        for (int y = 1; y < RD_GROUPS; ++y) t += sums[y][tx];
        if (i == kParams)
            stats[0] = t;
        else
            grad[i] = t;
    }
}

__device__ __forceinline__ bool structural_zero(int i) {
    return (i < ob1 && (i % kFeat) >= 24) || (i >= oW3 && i < ob3 && (i - oW3) / kHid >= 3) || (i >= ob3 && i - ob3 >= 3);
}

__global__ void mlp_adam_kernel(const float* __restrict__ grad, float* __restrict__ p32, float* __restrict__ m1,
                                float* __restrict__ m2, unsigned short* __restrict__ w16, float lr, float beta1,
                                float beta2, float eps, float bc1, float bc2) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    float p = p32[i];
    if (structural_zero(i)) {
        p = 0.0f;
        m1[i] = 0.0f;
        m2[i] = 0.0f;
    } else {
        const float gsum = grad[i];
        const float a = beta1 * m1[i] + (1.0f - beta1) * gsum;
        const float b = beta2 * m2[i] + (1.0f - beta2) * (gsum * gsum);
        m1[i] = a;
        m2[i] = b;
        p = p - lr * ((a / bc1) / (sqrtf(b / bc2) + eps));
    }
    p32[i] = p;
    if (i < ob1) w16[qW1 + (i - oW1)] = f2bf(p);
    else if (i >= oW2 && i < ob2) w16[qW2 + (i - oW2)] = f2bf(p);
    else if (i >= oW3 && i < ob3) w16[qW3 + (i - oW3)] = f2bf(p);
}

__global__ void mlp_sync_bf16_kernel(const float* __restrict__ p32, unsigned short* __restrict__ w16) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    if (i < ob1) w16[qW1 + (i - oW1)] = f2bf(p32[i]);
    else if (i >= oW2 && i < ob2) w16[qW2 + (i - oW2)] = f2bf(p32[i]);
    else if (i >= oW3 && i < ob3) w16[qW3 + (i - oW3)] = f2bf(p32[i]);
}

}  // namespace sx

using namespace sx;

extern "C" int sx_mlp_param_count(void) { return kParams; }
extern "C" int sx_mlp_bf16_count(void) { return kW16; }

extern "C" int sx_warm_features(const float* x4, const float* y4, const float* c4, const float* fixed,
                                const int* adj_ptr, const int* adj, const float* Lref, int n_verts, float gx, float gy,
                                float gz, float dt, void* feat, float* y_pred4, void* stream) {
    SX_REQUIRE(n_verts >= 0, "sx_warm_features: n_verts < 0");
    if (n_verts == 0) return SX_OK;
    SX_REQUIRE(x4 && y4 && c4 && fixed && adj_ptr && adj && Lref && feat, "sx_warm_features: null pointer");
    launch(warm_features_kernel, grid_for(n_verts, 256), 256, 0, as_stream(stream), n_verts, (const float4*)x4,
           (const float4*)y4, (const float4*)c4, fixed, adj_ptr, (const int2*)adj, Lref, gx, gy, gz, dt,
           (unsigned short*)feat, (float4*)y_pred4);
    return check_launch("warm_features_kernel");
}

extern "C" int sx_warm_apply(const float* y_pred4, const float* out4, const float* fixed, const float* Lref,
                             int n_verts, float* y4, void* stream) {
    SX_REQUIRE(n_verts >= 0, "sx_warm_apply: n_verts < 0");
    if (n_verts == 0) return SX_OK;
    SX_REQUIRE(y_pred4 && out4 && fixed && Lref && y4, "sx_warm_apply: null pointer");
    launch(warm_apply_kernel, grid_for(n_verts, 256), 256, 0, as_stream(stream), n_verts, (const float4*)y_pred4,
           out4, fixed, Lref, (float4*)y4);
    return check_launch("warm_apply_kernel");
}

extern "C" int sx_warm_record(const float* y4, const float* y_pred4, const float* fixed, const float* Lref,
                              int n_verts, float* c4, float* target4, void* stream) {
    SX_REQUIRE(n_verts >= 0, "sx_warm_record: n_verts < 0");
    if (n_verts == 0) return SX_OK;
    SX_REQUIRE(y4 && y_pred4 && fixed && Lref && c4, "sx_warm_record: null pointer");
    launch(warm_record_kernel, grid_for(n_verts, 256), 256, 0, as_stream(stream), n_verts, (const float4*)y4,
           (const float4*)y_pred4, fixed, Lref, (float4*)c4, (float4*)target4);
    return check_launch("warm_record_kernel");
}

extern "C" int sx_warm_select(const double* res_warm3, const double* res_cold3, const float* y_pred4, float* y4,
                              int n_verts, int* flags2, void* stream) {
    SX_REQUIRE(n_verts > 0, "sx_warm_select: n_verts must be positive");
    SX_REQUIRE(res_warm3 && res_cold3 && y_pred4 && y4 && flags2, "sx_warm_select: null pointer");
    launch(warm_select_kernel, grid_for(n_verts, 256), 256, 0, as_stream(stream), n_verts, res_warm3, res_cold3,
           (const float4*)y_pred4, (float4*)y4, flags2);
    return check_launch("warm_select_kernel");
}

extern "C" int sx_mlp_forward_tc(const void* feat, int n_rows, const void* w16, const float* p32, float* out4,
                                 int* status, void* stream) {
    SX_REQUIRE(n_rows >= 0, "sx_mlp_forward_tc: n_rows < 0");
    if (n_rows == 0) return SX_OK;
    SX_REQUIRE(feat && w16 && p32 && out4 && status, "sx_mlp_forward_tc: null pointer");
    const long long tiles = ((long long)n_rows + TC_ROWS - 1) / TC_ROWS;
    int dev = 0, sms = 0;
    SX_CUDA(cudaGetDevice(&dev));
    SX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // at most 7 CTAs fit an SM's shared memory, whose tensor memory holds 8: no
    // CTA waits in tcgen05.alloc
    const long long most = (long long)TC_PER_SM * sms;
    launch(mlp_forward_tc_kernel, (int)(tiles < most ? tiles : most), TC_THREADS, 0, as_stream(stream), n_rows,
           (const unsigned short*)feat, (const unsigned short*)w16, p32, out4, status);
    return check_launch("mlp_forward_tc_kernel");
}

extern "C" int sx_mlp_forward(const void* feat, int n_rows, const void* w16, const float* p32, float* out4,
                              void* stream) {
    SX_REQUIRE(n_rows >= 0, "sx_mlp_forward: n_rows < 0");
    if (n_rows == 0) return SX_OK;
    SX_REQUIRE(feat && w16 && p32 && out4, "sx_mlp_forward: null pointer");
    const int tiles = (n_rows + 15) / 16;
    int blocks = (tiles + MLP_BLOCK / 32 - 1) / (MLP_BLOCK / 32);
    if (blocks > 152 * 16) blocks = 152 * 16;
    launch(mlp_forward_kernel, blocks, MLP_BLOCK, 0, as_stream(stream), n_rows, (const unsigned short*)feat,
           (const unsigned short*)w16, p32, out4);
    return check_launch("mlp_forward_kernel");
}

// Training workspace: a partial of kPart floats per block, then the gradient.
static int train_blocks(int M) {
    const long long tiles = ((long long)M + TR_ROWS - 1) / TR_ROWS, most = 152LL * TR_PER_SM;
    return (int)(tiles < most ? tiles : most);
}

extern "C" size_t sx_mlp_train_workspace_bytes(int max_rows) {
    return ((size_t)train_blocks(max_rows > 0 ? max_rows : 1) * kPart + kParams) * 4 + 256;
}

static int mlp_grad_launches(float* part, const void* feat, const float* target4, const int* idx, int n_rows,
                             int n_valid, const void* w16, const float* p32, float* grad, float* stats,
                             cudaStream_t s) {
    SX_CUDA(cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(TrainSmem)));
    const int blocks = train_blocks(n_rows);
    launch(mlp_train_kernel, blocks, MLP_BLOCK, sizeof(TrainSmem), s, n_rows, idx, (const unsigned short*)feat,
           (const float4*)target4, 1.0f / (float)n_valid, (const unsigned short*)w16, p32, part);
    int rc = check_launch("mlp_train_kernel");
    if (rc) return rc;
    launch(mlp_reduce_kernel, (kPart + 31) / 32, 32 * RD_GROUPS, 0, s, blocks, (const float*)part, grad, stats);
    return check_launch("mlp_reduce_kernel");
}

extern "C" int sx_mlp_gradients(const void* feat, const float* target4, const int* idx, int n_rows, int n_valid,
                                const void* w16, const float* p32, float* grad, float* stats, void* ws,
                                size_t ws_bytes, void* stream) {
    SX_REQUIRE(n_rows > 0 && n_valid > 0, "sx_mlp_gradients: bad sizes");
    SX_REQUIRE(feat && target4 && idx && w16 && p32 && grad && stats && ws, "sx_mlp_gradients: null pointer");
    SX_REQUIRE(ws_bytes >= sx_mlp_train_workspace_bytes(n_rows), "sx_mlp_gradients: workspace too small");
    return mlp_grad_launches((float*)ws, feat, target4, idx, n_rows, n_valid, w16, p32, grad, stats, as_stream(stream));
}

extern "C" int sx_mlp_train_step(const void* feat, const float* target4, const int* idx, int n_rows, int n_valid,
                                 void* w16, float* p32, float* adam_m, float* adam_v, float lr, float beta1,
                                 float beta2, float eps, int step, float* stats, void* ws, size_t ws_bytes,
                                 void* stream) {
    SX_REQUIRE(n_rows > 0 && n_valid > 0 && step >= 1, "sx_mlp_train_step: bad sizes");
    SX_REQUIRE(feat && target4 && idx && w16 && p32 && adam_m && adam_v && stats && ws,
               "sx_mlp_train_step: null pointer");
    SX_REQUIRE(ws_bytes >= sx_mlp_train_workspace_bytes(n_rows), "sx_mlp_train_step: workspace too small");
    cudaStream_t s = as_stream(stream);
    float* grad = (float*)ws + (size_t)train_blocks(n_rows) * kPart;
    int rc = mlp_grad_launches((float*)ws, feat, target4, idx, n_rows, n_valid, w16, p32, grad, stats, s);
    if (rc) return rc;
    const float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
    launch(mlp_adam_kernel, grid_for(kParams, 256), 256, 0, s, (const float*)grad, p32, adam_m, adam_v,
           (unsigned short*)w16, lr, beta1, beta2, eps, bc1, bc2);
    return check_launch("mlp_adam_kernel");
}

extern "C" int sx_mlp_sync_bf16(const float* p32, void* w16, void* stream) {
    SX_REQUIRE(p32 && w16, "sx_mlp_sync_bf16: null pointer");
    launch(mlp_sync_bf16_kernel, grid_for(kParams, 256), 256, 0, as_stream(stream), p32, (unsigned short*)w16);
    return check_launch("mlp_sync_bf16_kernel");
}
