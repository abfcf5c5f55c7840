// LBVH broad phase: Morton codes, stable LSD radix sort, Karras 2012 hierarchy,
// single-launch bottom-up refit and stack traversal, for the reference's 32^3
// cell-grid BVH (framework/collision/lbvh_cell.py, class LBVH_CELL) and for a
// face-level LBVH over triangle soups.
#include <cuda/atomic>
#include <mutex>

#include "sx_common.cuh"
#include "sx_per_device.h"

namespace sx {

// ---------------------------------------------------------------------------
// Morton codes (lbvh_cell.py:87-102, :139-148)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long expand_bits(unsigned long long v) {
    v = (v | (v << 16)) & 0x030000FFull;
    v = (v | (v << 8)) & 0x0300F00Full;
    v = (v | (v << 4)) & 0x030C30C3ull;
    v = (v | (v << 2)) & 0x09249249ull;
    return v;
}
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
__device__ __forceinline__ unsigned morton3d(float x, float y, float z) {
    x = clampf(x * 1024.0f, 0.0f, 1023.0f);
    y = clampf(y * 1024.0f, 0.0f, 1023.0f);
    z = clampf(z * 1024.0f, 0.0f, 1023.0f);
    unsigned long long xx = expand_bits((unsigned long long)x), yy = expand_bits((unsigned long long)y),
                       zz = expand_bits((unsigned long long)z);
    return (unsigned)(xx | (yy << 1) | (zz << 2));
}
__device__ __forceinline__ unsigned morton_of(V3 p, V3 lo, V3 hi) {
    float x = (p.x - lo.x) / (hi.x - lo.x);
    float y = (p.y - lo.y) / (hi.y - lo.y);
    float z = (p.z - lo.z) / (hi.z - lo.z);
    return morton3d(clampf(x, 0.f, 1.f), clampf(y, 0.f, 1.f), clampf(z, 0.f, 1.f));
}

__device__ __forceinline__ V3 cell_size_of(const float* box6) {
    return V3{(box6[3] - box6[0]) / (float)kGridRes, (box6[4] - box6[1]) / (float)kGridRes,
              (box6[5] - box6[2]) / (float)kGridRes};
}
// assign_cell_centers (lbvh_cell.py:105-120)
__device__ __forceinline__ V3 cell_center(int i, V3 cs, V3 lo) {
    int x0 = i / (kGridRes * kGridRes), y0 = (i % (kGridRes * kGridRes)) / kGridRes, z0 = i % kGridRes;
    V3 p{cs.x * (float)x0 + 0.5f * cs.x, cs.y * (float)y0 + 0.5f * cs.y, cs.z * (float)z0 + 0.5f * cs.z};
    return add(p, lo);
}

__global__ void cell_morton_kernel(unsigned* codes, int* ids) {
    pdl_entry();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kNumCells) return;
    const float box[6] = {0.f, 0.f, 0.f, 1e3f, 1e3f, 1e3f};
    V3 lo{0.f, 0.f, 0.f}, hi{1e3f, 1e3f, 1e3f};
    V3 cs = cell_size_of(box);
    codes[i] = morton_of(cell_center(i, cs, lo), lo, hi);
    ids[i] = i;
}

__global__ void face_morton_kernel(int F, const float4* __restrict__ mn4, const float4* __restrict__ mx4,
                                   const float* __restrict__ box6, unsigned* codes, int* ids) {
    pdl_entry();
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    V3 lo{box6[0], box6[1], box6[2]}, hi{box6[3], box6[4], box6[5]};
    V3 c = scale(0.5f, add(mk(mx4[f]), mk(mn4[f])));
    codes[f] = morton_of(c, lo, hi);
    ids[f] = f;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort, 8-bit digits.  Few pairs take rs_cluster_kernel, more
// three launches a digit:
//   upsweep : per-tile digit histogram -> hist[digit * nblocks + block]
//   scan    : one block per digit scans its column (exclusive over the tiles,
//             in tile order) and writes the digit's total
//   scatter : each tile takes its digit bases (exclusive scan of the 256
//             totals + its column offset); each warp owns a contiguous 256-key
//             slice of the tile and ranks its keys within their digit in input
//             order (__match_any_sync, warp-private counters), so the order is
//             stable with three block barriers per tile.
// ---------------------------------------------------------------------------
constexpr int RS_BLOCK = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_BLOCK * RS_ITEMS;
constexpr int RS_WARPS = RS_BLOCK / 32;

__global__ void __launch_bounds__(RS_BLOCK) rs_upsweep(const unsigned* __restrict__ keys, int n, int shift,
                                                       unsigned dmask, unsigned* __restrict__ hist, int nblocks) {
    pdl_entry();
    __shared__ unsigned cnt[256];
    const int tid = threadIdx.x;
    cnt[tid] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * RS_TILE;
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        long long idx = base + r * RS_BLOCK + tid;
        if (idx < n) atomicAdd(&cnt[(keys[idx] >> shift) & dmask], 1u);
    }
    __syncthreads();
    hist[(size_t)tid * nblocks + blockIdx.x] = cnt[tid];
}

// Exclusive scan of one value per thread over a 256-thread block; returns the
// block total through *total.
__device__ __forceinline__ unsigned block256_excl_scan(unsigned v, unsigned* total) {
    __shared__ unsigned wsum[RS_WARPS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < RS_WARPS; ++k) {
        before += k < w ? wsum[k] : 0u;
        all += wsum[k];
    }
    __syncthreads();
    *total = all;
    return before + incl - v;
}

// Block d: exclusive scan of hist[d * nblocks .. (d + 1) * nblocks) in place,
// the column total to tot[d].
__global__ void __launch_bounds__(RS_BLOCK) rs_digit_scan(unsigned* __restrict__ hist, int nblocks,
                                                          unsigned* __restrict__ tot) {
    pdl_entry();
    unsigned* col = hist + (size_t)blockIdx.x * nblocks;
    unsigned carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += RS_BLOCK) {
        const int b = b0 + threadIdx.x;
        const unsigned v = b < nblocks ? col[b] : 0u;
        unsigned sum;
        const unsigned ex = block256_excl_scan(v, &sum);
        if (b < nblocks) col[b] = carry + ex;
        carry += sum;
    }
    if (threadIdx.x == 0) tot[blockIdx.x] = carry;
}

// Single-block scan over n entries (exclusive or inclusive), 1024 threads, in
// segments of 32768 staged in (dynamic) shared memory: one coalesced load of
// the segment, each thread sums 32 consecutive entries (one padding word per
// 32 keeps those reads on distinct banks), a block scan of the sums (warp
// shuffles, then the 32 warp totals), each thread rewrites its 32, one
// coalesced store; the running total carries into the next segment.
constexpr int SCAN_SEG = 32768;
constexpr int SCAN_PER = SCAN_SEG / 1024;
constexpr size_t SCAN_SMEM = (size_t)(SCAN_SEG + SCAN_SEG / 32) * 4;

__device__ __forceinline__ int scan_slot(int i) { return i + (i >> 5); }

__global__ void __launch_bounds__(1024) scan_single_block(unsigned* data, int n, int inclusive) {
    pdl_entry();
    extern __shared__ unsigned seg[];
    __shared__ unsigned wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned carry = 0;
    for (int s0 = 0; s0 < n; s0 += SCAN_SEG) {
        const int m = min(SCAN_SEG, n - s0);
#pragma unroll 8
        for (int i = tid; i < SCAN_SEG; i += 1024) seg[scan_slot(i)] = i < m ? data[s0 + i] : 0u;
        __syncthreads();
        unsigned sum = 0;
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k) sum += seg[scan_slot(tid * SCAN_PER + k)];
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        unsigned before = 0, total = 0;
        for (int k = 0; k < 32; ++k) {
            before += k < w ? wsum[k] : 0u;
            total += wsum[k];
        }
        unsigned run = carry + before + incl - sum;
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k) {
            const int j = scan_slot(tid * SCAN_PER + k);
            const unsigned x = seg[j];
            seg[j] = inclusive ? run + x : run;
            run += x;
        }
        __syncthreads();
#pragma unroll 8
        for (int i = tid; i < m; i += 1024) data[s0 + i] = seg[scan_slot(i)];
        carry += total;
        __syncthreads();
    }
}

// The shared-memory limit is raised once per device.
static cudaError_t scan_smem_attr() {
    static PerDevice attr;
    int dev = -1;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return (cudaError_t)attr.get(dev, [] {
        return (int)cudaFuncSetAttribute(scan_single_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)SCAN_SMEM);
    });
}

static int launch_scan_single_block(unsigned* data, int n, int inclusive, cudaStream_t s) {
    const cudaError_t attr = scan_smem_attr();
    if (attr != cudaSuccess) return cuda_status(attr, "cudaFuncSetAttribute(scan_single_block)");
    launch(scan_single_block, 1, 1024, SCAN_SMEM, s, data, n, inclusive);
    return check_launch("scan_single_block");
}

__global__ void __launch_bounds__(RS_BLOCK) rs_scatter(const unsigned* __restrict__ kin,
                                                       const int* __restrict__ vin, unsigned* __restrict__ kout,
                                                       int* __restrict__ vout, int n, int shift, unsigned dmask,
                                                       const unsigned* __restrict__ hist,
                                                       const unsigned* __restrict__ tot, int nblocks) {
    pdl_entry();
    __shared__ unsigned s_off[RS_WARPS][256];
    __shared__ unsigned s_gbase[256], s_lbase[256];
    __shared__ unsigned s_key[RS_TILE];
    __shared__ int s_val[RS_TILE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned all;
    const unsigned digit_base = block256_excl_scan(tot[tid], &all) + hist[(size_t)tid * nblocks + blockIdx.x];
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) s_off[w][tid] = 0;
    __syncthreads();
    // warp `warp` owns keys [tile + warp * 256, tile + (warp + 1) * 256)
    const long long tile = (long long)blockIdx.x * RS_TILE;
    const long long base = tile + warp * (RS_ITEMS * 32);
    unsigned key[RS_ITEMS], rank[RS_ITEMS];
    int val[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const long long idx = base + r * 32 + lane;
        key[r] = idx < n ? kin[idx] : 0u;
        val[r] = idx < n ? vin[idx] : 0;
    }
    unsigned* cnt = s_off[warp];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        const bool valid = base + r * 32 + lane < n;
        const unsigned digit = valid ? ((key[r] >> shift) & dmask) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, digit);
        const unsigned before = valid ? cnt[digit] : 0u;
        rank[r] = before + __popc(peers & lt_mask);
        __syncwarp();
        if (valid && (__ffs(peers) - 1) == lane) cnt[digit] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: the tile's count, its offset in the tile's digit order, and
    // each warp's offset within it
    unsigned tsum = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) tsum += s_off[w][tid];
    const unsigned lbase = block256_excl_scan(tsum, &all);
    s_lbase[tid] = lbase;
    s_gbase[tid] = digit_base;
    unsigned run = lbase;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const unsigned c = s_off[w][tid];
        s_off[w][tid] = run;
        run += c;
    }
    __syncthreads();
    // the tile in digit order (stable within a digit) in shared memory ...
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
        if (base + r * 32 + lane < n) {
            const unsigned lp = cnt[(key[r] >> shift) & dmask] + rank[r];
            s_key[lp] = key[r];
            s_val[lp] = val[r];
        }
    }
    __syncthreads();
    // ... written out so that consecutive threads fill consecutive slots of
    // each digit's run
    const int count = (int)min((long long)RS_TILE, (long long)n - tile);
    for (int i = tid; i < count; i += RS_BLOCK) {
        const unsigned k = s_key[i];
        const unsigned d = (k >> shift) & dmask;
        const unsigned g = s_gbase[d] + ((unsigned)i - s_lbase[d]);
        kout[g] = k;
        vout[g] = s_val[i];
    }
}

// All passes of a sort of at most 65 536 pairs in one launch: the tiles of one
// cluster of up to 16 blocks, 1024 x ITEMS pairs each.  A pass ranks the tile's
// keys as rs_scatter does, publishes the tile's digit counts in shared memory,
// and takes its digit bases from all tiles' counts (distributed shared memory)
// where the kernels above go through two launches; the pairs then go to their
// places in the same arrays, which every tile has read by then.  What bounds it
// is the chain of barriers and round trips, about 5 us a pass of small tiles, against
// 9 us for the three launches; the line is where the few SMs' ranking and writing take
// over.  15 / 30 bits, three launches a pass -> one in all: 7938 pairs 18.8 -> 10.3 /
// 35.7 -> 19.3 us, 20 011 22.0 -> 13.7 / 47.4 -> 25.8, 65 000 18.0 -> 16.4 /
// 38.9 -> 37.1; with 8 pairs a thread, 100 000: 16.3 -> 22.7 / 37.2 -> 60.3.
constexpr int RC_BLOCK = 1024, RC_WARPS = RC_BLOCK / 32, RC_CLUSTER = 16, RC_MAX_ITEMS = 4;
constexpr size_t rc_smem(int items) { return (size_t)(RC_WARPS * 256 + 2 * RC_BLOCK * items) * 4; }

// Exclusive scan of one value per thread over the first 256 threads of the block
// (the others pass 0 and get the total).
__device__ __forceinline__ unsigned first256_excl_scan(unsigned v, unsigned* wsum) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (w < 8 && lane == 31) wsum[w] = incl;
    __syncthreads();
    unsigned before = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) before += k < w ? wsum[k] : 0u;
    __syncthreads();
    return before + incl - v;
}

template <int ITEMS>
__global__ void __launch_bounds__(RC_BLOCK, 1) rs_cluster_kernel(unsigned* keys, int* vals, int n, int first, int bits) {
    pdl_entry();
    constexpr int TILE = RC_BLOCK * ITEMS;
    extern __shared__ unsigned dyn[];
    unsigned(*s_off)[256] = reinterpret_cast<unsigned(*)[256]>(dyn);
    unsigned* s_key = dyn + RC_WARPS * 256;
    int* s_val = reinterpret_cast<int*>(s_key + TILE);
    __shared__ unsigned s_count[256], s_gbase[256], s_lbase[256], s_wsum[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tiles = gridDim.x, tile = blockIdx.x;  // the grid is one cluster
    const unsigned lt_mask = (1u << lane) - 1u;
    const int start = tile * TILE, count = min(max(n - start, 0), TILE);
    const int base = warp * (ITEMS * 32) + lane;
    unsigned* cnt = s_off[warp];
    for (int shift = first; shift < first + bits; shift += 8) {
        const int width = min(first + bits - shift, 8);
        const unsigned dmask = (1u << width) - 1u;
        unsigned key[ITEMS], rank[ITEMS];
        int val[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int i = base + r * 32;  // written by other blocks in the last pass: not from L1
            key[r] = i < count ? __ldcg(keys + start + i) : 0u;
            val[r] = i < count ? __ldcg(vals + start + i) : 0;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) cnt[k * 32 + lane] = 0u;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const bool valid = base + r * 32 < count;
            const unsigned digit = valid ? ((key[r] >> shift) & dmask) : 256u;
            const unsigned peers = __match_any_sync(0xffffffffu, digit);
            const unsigned before = valid ? cnt[digit] : 0u;
            rank[r] = before + __popc(peers & lt_mask);
            __syncwarp();
            if (valid && (__ffs(peers) - 1) == lane) cnt[digit] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        unsigned sum = 0u;
        if (tid < 256) {
#pragma unroll 8
            for (int w = 0; w < RC_WARPS; ++w) sum += s_off[w][tid];
            s_count[tid] = sum;
        }
        const unsigned lbase = first256_excl_scan(sum, s_wsum);
        if (tid < 256) {
            s_lbase[tid] = lbase;
            unsigned run = lbase;
#pragma unroll 8
            for (int w = 0; w < RC_WARPS; ++w) {
                const unsigned c = s_off[w][tid];
                s_off[w][tid] = run;
                run += c;
            }
        }
        cluster_barrier();  // all tiles' counts published, all their pairs read
        unsigned before = 0u, all = 0u;
        if (tid < 256) {
            unsigned c[RC_CLUSTER];
#pragma unroll
            for (int t = 0; t < RC_CLUSTER; ++t) c[t] = t < tiles ? load_cluster(s_count + tid, t) : 0u;
#pragma unroll
            for (int t = 0; t < RC_CLUSTER; ++t) {
                before += t < tile ? c[t] : 0u;
                all += c[t];
            }
        }
        const unsigned digit_base = first256_excl_scan(all, s_wsum);
        if (tid < 256) s_gbase[tid] = digit_base + before;
        // the tile in digit order, then consecutive threads to consecutive places
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            if (base + r * 32 < count) {
                const unsigned lp = cnt[(key[r] >> shift) & dmask] + rank[r];
                s_key[lp] = key[r];
                s_val[lp] = val[r];
            }
        }
        __syncthreads();
        for (int i = tid; i < count; i += RC_BLOCK) {
            const unsigned k = s_key[i];
            const unsigned d = (k >> shift) & dmask;
            const unsigned g = s_gbase[d] + ((unsigned)i - s_lbase[d]);
            keys[g] = k;
            vals[g] = s_val[i];
        }
        cluster_barrier();  // the pass is written, and no block leaves while its counts are read
    }
}

using ClusterSort = void (*)(unsigned*, int*, int, int, int);
static ClusterSort cluster_sort_kernel(int items) {
    return items == 1 ? rs_cluster_kernel<1> : items == 2 ? rs_cluster_kernel<2>
                                           : rs_cluster_kernel<RC_MAX_ITEMS>;
}
// Largest cluster of the sort that the current device can hold, 0 for none.  The
// kernels' limits are raised once per device.
static int cluster_sort_blocks() {
    static PerDevice blocks;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return blocks.get(dev, [] {
        for (int items = 1; items <= RC_MAX_ITEMS; items *= 2) {
            const ClusterSort k = cluster_sort_kernel(items);
            if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rc_smem(items)) !=
                    cudaSuccess ||
                cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
                cudaGetLastError();
                return 0;
            }
        }
        for (int c = RC_CLUSTER; c >= 8; c /= 2) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim = {(unsigned)c, 1, 1};
            cfg.gridDim = c;
            cfg.blockDim = RC_BLOCK;
            cfg.dynamicSmemBytes = rc_smem(RC_MAX_ITEMS);
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int active = 0;
            if (cudaOccupancyMaxActiveClusters(&active, rs_cluster_kernel<RC_MAX_ITEMS>, &cfg) == cudaSuccess &&
                active > 0)
                return c;
            cudaGetLastError();
        }
        return 0;
    });
}

int scan_u32(unsigned* data, int n, int inclusive, cudaStream_t s) {
    if (n <= 0) return SX_OK;
    return launch_scan_single_block(data, n, inclusive, s);
}

static inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
static inline int rs_nblocks(int n) { return n <= 0 ? 1 : (n + RS_TILE - 1) / RS_TILE; }
static size_t rs_ws_bytes(int n) {
    size_t nn = (size_t)(n > 0 ? n : 1);
    return align256(nn * 4) * 2 + align256((size_t)256 * rs_nblocks(n) * 4) + align256(256 * 4);
}

static int radix_sort(unsigned* keys, int* vals, int n, int bits, void* ws, size_t ws_bytes, cudaStream_t s,
                      int first = 0) {
    SX_REQUIRE(bits >= 1 && first >= 0 && first + bits <= 32, "radix sort: bits must be in [1, 32]");
    if (n <= 1) return SX_OK;
    SX_REQUIRE(ws && ws_bytes >= rs_ws_bytes(n), "radix sort: workspace too small (%zu < %zu)", ws_bytes,
               rs_ws_bytes(n));
    char* p = (char*)ws;
    unsigned* kalt = (unsigned*)p;
    p += align256((size_t)n * 4);
    int* valt = (int*)p;
    p += align256((size_t)n * 4);
    unsigned* hist = (unsigned*)p;
    const int nb = rs_nblocks(n);
    p += align256((size_t)256 * nb * 4);
    unsigned* tot = (unsigned*)p;
    const int passes = (bits + 7) / 8;
    const int tiles = cluster_sort_blocks();  // a cluster of fewer blocks, fewer pairs
    if (n <= tiles * RC_BLOCK * RC_MAX_ITEMS) {
        int items = 1, blocks = 1;
        while (items < RC_MAX_ITEMS && n > tiles * RC_BLOCK * items) items *= 2;
        while (blocks * RC_BLOCK * items < n) blocks *= 2;
        launch_cluster(cluster_sort_kernel(items), blocks, RC_BLOCK, rc_smem(items), s, keys, vals, n, first, bits);
        return check_launch("rs_cluster_kernel");
    }
    unsigned* ki = keys;
    int* vi = vals;
    unsigned* ko = kalt;
    int* vo = valt;
    for (int pass = 0; pass < passes; ++pass) {
        const int shift = first + 8 * pass;
        // the last digit keeps only the key bits below `first + bits`: the other
        // bits ride along unsorted
        const int width = bits - 8 * pass < 8 ? bits - 8 * pass : 8;
        const unsigned dmask = (1u << width) - 1u;
        launch(rs_upsweep, nb, RS_BLOCK, 0, s, ki, n, shift, dmask, hist, nb);
        launch(rs_digit_scan, 256, RS_BLOCK, 0, s, hist, nb, tot);
        launch(rs_scatter, nb, RS_BLOCK, 0, s, ki, vi, ko, vo, n, shift, dmask, (const unsigned*)hist,
               (const unsigned*)tot, nb);
        unsigned* tk = ki; ki = ko; ko = tk;
        int* tv = vi; vi = vo; vo = tv;
    }
    if (ki != keys) {
        SX_CUDA(cudaMemcpyAsync(keys, ki, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
        SX_CUDA(cudaMemcpyAsync(vals, vi, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
    }
    return check_launch("radix_sort");
}

// ---------------------------------------------------------------------------
// Karras 2012 hierarchy (lbvh_cell.py:256-336, :384-430)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int kdelta(int i, long long j, int n, const unsigned* c, int tie) {
    if (j > n - 1 || j < 0) return -1;
    unsigned x = c[i] ^ c[(int)j];
    if (x == 0) return tie ? 32 + __clz(i ^ (int)j) : 32;
    return __clz(x);
}

__global__ void karras_kernel(int n, const unsigned* __restrict__ c, int tie, int* child_a, int* child_b,
                              int* range_l, int* range_r, int* parent) {
    pdl_entry();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) parent[0] = -1;
    if (i >= n - 1) return;
    // determine_range
    int dl = kdelta(i, (long long)i - 1, n, c, tie), dr = kdelta(i, (long long)i + 1, n, c, tie);
    int d = 1, dmin = dl;
    if (dr < dl) { d = -1; dmin = dr; }
    long long lmax = 2;
    while (lmax < 4LL * n && kdelta(i, (long long)i + lmax * d, n, c, tie) > dmin) lmax <<= 2;
    long long l = 0;
    for (long long t = lmax / 2; t > 0; t /= 2) {
        long long j = (long long)i + (l + t) * d;
        int dd = (j >= 0 && j < n) ? kdelta(i, j, n, c, tie) : -1;
        if (dd > dmin) l += t;
    }
    int s = i, e = (int)(i + l * d);
    if (d == -1) { s = (int)(i + l * d); e = i; }
    // find_split
    int split;
    if (c[s] == c[e] && !tie) {
        split = (s + e) / 2;
    } else {
        int common = kdelta(s, e, n, c, tie);
        split = s;
        int step = e - s;
        while (step > 1) {
            step = (step + 1) / 2;
            int ns = split + step;
            if (ns < e && kdelta(s, ns, n, c, tie) > common) split = ns;
        }
    }
    int left = split, right = split + 1;
    if (split == s) left += n - 1;
    if (right == e) right += n - 1;
    child_a[i] = left;
    child_b[i] = right;
    range_l[i] = s;
    range_r[i] = e;
    parent[left] = i;
    parent[right] = i;
}

// ---------------------------------------------------------------------------
// Cell-grid BVH build (LBVH_CELL.build, lbvh_cell.py:637-653)
// ---------------------------------------------------------------------------
// box_out (optional): a copy of box6.
__global__ void face_cell_kernel(int F, const float4* __restrict__ mn4, const float4* __restrict__ mx4,
                                 const float* box6, float* box_out, unsigned* keys, int* ids, float* grid8) {
    pdl_entry();
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    V3 lo{box6[0], box6[1], box6[2]};
    V3 cs = cell_size_of(box6);
    if (f == 0) {
        grid8[0] = cs.x;
        grid8[1] = cs.y;
        grid8[2] = cs.z;
        grid8[3] = grid8[4] = grid8[5] = 0.0f;  // max leaf overhang, raised by the leaf kernel
        grid8[6] = grid8[7] = 0.0f;             // [7]: the leaf kernel's blocks that are done
    }
    if (box_out != nullptr && f < 6) box_out[f] = box6[f];
    if (f >= F) return;
    V3 c = scale(0.5f, add(mk(mn4[f]), mk(mx4[f])));
    int ix = min(max(f2i_sat((c.x - lo.x) / cs.x), 0), kGridRes - 1);
    int iy = min(max(f2i_sat((c.y - lo.y) / cs.y), 0), kGridRes - 1);
    int iz = min(max(f2i_sat((c.z - lo.z) / cs.z), 0), kGridRes - 1);
    keys[f] = (unsigned)(ix * kGridRes * kGridRes + iy * kGridRes + iz);
    ids[f] = f;
}

// prefix[c] = faces in cells 0 .. c, from the sorted cells: thread i writes the
// cells from key i - 1 up to key i (to the end for the last), a long run of empty
// cells with its whole warp.  No counters to clear, raise and scan.
__global__ void __launch_bounds__(256) cell_bounds_kernel(int F, const unsigned* __restrict__ keys,
                                                          int* __restrict__ prefix) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    int from = 0, to = 0;
    if (i <= F) {
        from = i == 0 ? 0 : (int)keys[i - 1];
        to = i == F ? kNumCells : (int)keys[i];
    }
    unsigned runs = __ballot_sync(0xffffffffu, to > from);
    for (; runs != 0u; runs &= runs - 1u) {
        const int l = __ffs(runs) - 1;
        const int end = __shfl_sync(0xffffffffu, to, l), n = i - lane + l;
        for (int c = __shfl_sync(0xffffffffu, from, l) + lane; c < end; c += 32) prefix[c] = n;
    }
}

// Node boxes are float4 pairs; min.w carries the node's face count (int bits)
// so that one 16-byte load gives a child's box corner and whether it is empty.
__device__ __forceinline__ void store_box(float4* nmin4, float4* nmax4, int i, V3 a, V3 b, int nf = 0) {
    nmin4[i] = make_float4(a.x, a.y, a.z, __int_as_float(nf));
    nmax4[i] = make_float4(b.x, b.y, b.z, 0.0f);
}
__device__ __forceinline__ V3 load_cg(const float4* p) {
    float4 v = __ldcg(p);
    return V3{v.x, v.y, v.z};
}

// assign_leaf_cell_nodes (:602-634) fused with a bottom-up refit that applies
// the rules of compute_cell_node_aabbs (:491-522).  The second thread to reach
// an internal node computes it from both (finished) children.  Each leaf also
// writes its faces' records (min.xyz + face id, max.xyz) in sorted order, the
// contiguous array the traversal scans.
// The cell tree is the perfect tree over the 32768 row-major cells (leaf slot
// i = cell i, child_a = lower half).  The Karras build numbers an internal
// node covering the aligned slot range [l, r] of size s >= 2 as 0 for the
// root, r when it is a left child (l / s even) and l when it is a right child;
// a leaf is slot + 32767.  The refit therefore needs no climbing: one block
// per z-column (32 leaves, an aligned subtree) fits its leaves and the
// subtree's 31 nodes in shared memory, and the last block to finish fits the 1023
// nodes above the columns level by level.
__device__ __forceinline__ int cell_node_index(int l, int size) {
    if (size == kNumCells) return 0;
    if (size == 1) return l + kNumCells - 1;
    return ((l / size) & 1) == 0 ? l + size - 1 : l;
}

struct NodeBox {
    V3 a, b;
    int n;
};
// compute_cell_node_aabbs (lbvh_cell.py:491-522): union of the non-empty
// children; two empty children give the point at the mean of their corners
__device__ __forceinline__ NodeBox join_nodes(const NodeBox& l, const NodeBox& r) {
    NodeBox o;
    if (l.n > 0 && r.n > 0) {
        o.a = vmin(l.a, r.a);
        o.b = vmax(l.b, r.b);
    } else if (l.n > 0) {
        o.a = l.a;
        o.b = l.b;
    } else if (r.n > 0) {
        o.a = r.a;
        o.b = r.b;
    } else {
        o.a = scale(0.25f, add(add(add(l.a, l.b), r.a), r.b));
        o.b = o.a;
    }
    o.n = l.n + r.n;
    return o;
}

// Block = one z-column (cells col*32 .. col*32+31); the 1024 columns fit one wave
// of blocks.  Most of a column's cells are empty: a lane each writes the centre
// point, and the warps take the cells that hold faces, two batches of 32 faces at
// once.  The last block to finish fits the 1023 nodes above the columns (sizes 64 ..
// 32768).  A chain of dependent loads (prefix, face, box) bounds it; a warp that
// took four cells one after the other went through it four times.  The whole
// build, with the sums before each cell read off the sorted cells instead of cleared,
// counted and scanned: 64 x 64 sheet 35.6 -> 26.5 us, 181 x 139 40.2 -> 29.1, 256 x
// 256 46.9 -> 35.2.
constexpr int kColumnRefitThreads = 256;

__global__ void __launch_bounds__(kColumnRefitThreads) cell_column_refit_kernel(
    const float* __restrict__ box6, const int* __restrict__ prefix, const int* __restrict__ sorted_face_ids,
    const float4* __restrict__ fmn4, const float4* __restrict__ fmx4, int* __restrict__ num_faces, float4* nmin4,
    float4* nmax4, float4* __restrict__ frec, float* grid8) {
    pdl_entry();
    __shared__ NodeBox tree[64];  // [32 + k]: leaf k; [16 + k], [8 + k], ...: levels above
    __shared__ NodeBox top[2 * kColumnRefitThreads];  // the same above the columns, from [256 + k] on
    __shared__ bool last;
    const int col = blockIdx.x, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const V3 lo{box6[0], box6[1], box6[2]};
    const V3 cs = cell_size_of(box6);
    // every warp: lane z's cell
    const int i = col * kGridRes + lane;
    const int rl = i == 0 ? 0 : prefix[i - 1];
    const int size = prefix[i] - rl;
    const unsigned occ = __ballot_sync(0xffffffffu, size > 0);
    if (w == 0 && size == 0) tree[32 + lane] = NodeBox{cell_center(i, cs, lo), cell_center(i, cs, lo), 0};
    unsigned todo = occ;
    for (int k = 0; todo != 0u; ++k, todo &= todo - 1u) {
        if (k % (kColumnRefitThreads / 32) != w) continue;
        const int z = __ffs(todo) - 1;
        const int first = __shfl_sync(0xffffffffu, rl, z), n = __shfl_sync(0xffffffffu, size, z);
        const V3 c = cell_center(col * kGridRes + z, cs, lo);
        V3 a = c, b = c;
        for (int j = lane; j < n; j += 64) {
            const bool two = j + 32 < n;
            const int f0 = sorted_face_ids[first + j], f1 = two ? sorted_face_ids[first + j + 32] : f0;
            const float4 a0 = fmn4[f0], b0 = fmx4[f0], a1 = fmn4[f1], b1 = fmx4[f1];
            a = vmin(vmin(a, mk(a0)), mk(a1));
            b = vmax(vmax(b, mk(b0)), mk(b1));
            frec[2 * (first + j)] = make_float4(a0.x, a0.y, a0.z, __int_as_float(f0));
            frec[2 * (first + j) + 1] = make_float4(b0.x, b0.y, b0.z, 0.0f);
            if (two) {
                frec[2 * (first + j + 32)] = make_float4(a1.x, a1.y, a1.z, __int_as_float(f1));
                frec[2 * (first + j + 32) + 1] = make_float4(b1.x, b1.y, b1.z, 0.0f);
            }
        }
        __syncwarp();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = vmin(a, V3{__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                           __shfl_xor_sync(0xffffffffu, a.z, o)});
            b = vmax(b, V3{__shfl_xor_sync(0xffffffffu, b.x, o), __shfl_xor_sync(0xffffffffu, b.y, o),
                           __shfl_xor_sync(0xffffffffu, b.z, o)});
        }
        if (lane == 0) tree[32 + z] = NodeBox{a, b, n};
    }
    __syncthreads();
    if (w == 0) {
        const NodeBox nb = tree[32 + lane];
        num_faces[i + kNumCells - 1] = nb.n;
        store_box(nmin4, nmax4, i + kNumCells - 1, nb.a, nb.b, nb.n);
        // how far this leaf's box reaches beyond its cell (>= 0), maximised over the
        // grid: the traversal scans the cells within that reach
        const int x0 = i / (kGridRes * kGridRes), y0 = (i % (kGridRes * kGridRes)) / kGridRes;
        const float clo[3] = {lo.x + cs.x * (float)x0, lo.y + cs.y * (float)y0, lo.z + cs.z * (float)lane};
        const float chi[3] = {lo.x + cs.x * (float)(x0 + 1), lo.y + cs.y * (float)(y0 + 1),
                              lo.z + cs.z * (float)(lane + 1)};
        const float am[3] = {nb.a.x, nb.a.y, nb.a.z}, bm[3] = {nb.b.x, nb.b.y, nb.b.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float ext = nb.n > 0 ? fmaxf(fmaxf(clo[k] - am[k], bm[k] - chi[k]), 0.0f) : 0.0f;
            const unsigned most = __reduce_max_sync(0xffffffffu, ext > 0.0f ? __float_as_uint(ext) : 0u);
            if (lane == 0 && most != 0u) atomicMax(reinterpret_cast<unsigned*>(grid8) + 3 + k, most);
        }
        // occupancy word of the column, and the column's subtree, level by level
        if (lane == 0) reinterpret_cast<unsigned*>(grid8)[kGridHeader + col] = occ;
        for (int half = 16, sz = 2; half >= 1; half >>= 1, sz <<= 1) {
            if (lane < half) {
                const NodeBox nb = join_nodes(tree[2 * half + 2 * lane], tree[2 * half + 2 * lane + 1]);
                tree[half + lane] = nb;
                const int node = cell_node_index(col * kGridRes + lane * sz, sz);
                num_faces[node] = nb.n;
                store_box(nmin4, nmax4, node, nb.a, nb.b, nb.n);
            }
            __syncwarp();
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) last = atomicAdd(reinterpret_cast<int*>(grid8) + 7, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int t = threadIdx.x;
    if (t == 0) grid8[7] = 0.0f;
    // four columns a thread, two levels in registers, the others in shared memory
    static_assert(4 * kColumnRefitThreads == kGridRes * kGridRes, "four columns a thread");
    auto put = [&](int l, int size, const NodeBox& nb) {
        const int node = cell_node_index(l, size);
        num_faces[node] = nb.n;
        store_box(nmin4, nmax4, node, nb.a, nb.b, nb.n);
    };
    NodeBox c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int node = cell_node_index((4 * t + k) * kGridRes, kGridRes);
        const float4 na = __ldcg(nmin4 + node), nb = __ldcg(nmax4 + node);
        c[k] = NodeBox{mk(na), mk(nb), __float_as_int(na.w)};
    }
    c[0] = join_nodes(c[0], c[1]);
    c[2] = join_nodes(c[2], c[3]);
    put(4 * t * kGridRes, 2 * kGridRes, c[0]);
    put((4 * t + 2) * kGridRes, 2 * kGridRes, c[2]);
    c[0] = join_nodes(c[0], c[2]);
    put(4 * t * kGridRes, 4 * kGridRes, c[0]);
    top[kColumnRefitThreads + t] = c[0];
    for (int half = kColumnRefitThreads / 2, sz = 8 * kGridRes; half >= 1; half >>= 1, sz <<= 1) {
        __syncthreads();
        if (t < half) {
            const NodeBox nb = join_nodes(top[2 * (half + t)], top[2 * (half + t) + 1]);
            top[half + t] = nb;
            put(t * sz, sz, nb);
        }
    }
}

// traverse_cell_bvh_single (lbvh_cell.py:662-714) as a walk over grid cells.
//
// The reference pops a node, skips it when empty or not overlapping, and
// otherwise scans a leaf's faces or pushes child_a then child_b.  The cell tree
// is always the perfect tree that the Karras build makes over the 32^3
// distinct cell codes, child_a covering the lower half of a node's leaf slots,
// and leaf slot i holds row-major cell i (lbvh_cell.py:604-634).  Its
// depth-first walk therefore reaches exactly the non-empty leaves whose boxes
// overlap the query (every ancestor of such a leaf contains its box), in
// descending slot = descending cell index.  A leaf's box is its cell grown by
// at most the build's maximum overhang (grid8[3..5]), so scanning the cells
// within that reach of the query box, in descending index, and applying the
// same leaf and face tests produces the same candidate list in the same order,
// with independent loads instead of a chain of dependent node fetches.
__device__ __forceinline__ void cell_range(float qa, float qb, float o, float c, float e, int* i0, int* i1) {
    // A leaf box lies within [o + c i - e, o + c (i + 1) + e] up to the
    // rounding of those bounds (relative 2^-24 of |o| + 64 c and of e); the
    // divisions below carry relative 2^-22 of (|q| + e + |o|) / c.  delta covers
    // both 64 times over, so a cell is left out only when no leaf box in it
    // can reach the query box.  A zero or non-finite cell size gives the full
    // range.
    const float delta = 1.5e-5f * ((fabsf(qa) + fabsf(qb) + 2.0f * e + 2.0f * fabsf(o) + 64.0f * c) / c);
    const float f0 = ceilf((qa - e - o) / c - 1.0f - delta), f1 = floorf((qb + e - o) / c + delta);
    *i0 = (int)fmaxf(f0, 0.0f);
    *i1 = (int)fminf(f1, (float)(kGridRes - 1));
}

// A warp takes one query after the other.  It walks the (x, y) columns of the query's cell
// range in descending order.  In each column, lane l takes cell z = 31 - l, so
// that ascending lanes are the reference's descending-z visiting order: the
// occupied cells' leaf boxes are tested at once, a warp scan lays the faces of
// the cells that pass end to end in that order, and the lanes test those faces
// 32 at a time (each lane finds its cell by a binary search over the scan).  A
// ballot places each overlapping face after those of lower lanes, so
// candidates come out in descending cell order and, within a cell, in sorted
// face order -- the reference's visiting order -- with every lane busy.
//
// Instruction issue bounds it (a thousand a query, 2.3 a cycle and SM, DRAM idle),
// so: the cell ranges' divisions are done once, an axis a lane; cells that pass
// with 20 faces or more on average (CT_LONG_CELL; a 256 x 256 sheet has 150) are
// scanned one after the other, which takes half the instructions per 32 faces of
// the search for each lane's cell (63 against 77 us, the crossing is flat between
// 12 and 20); empty runs of columns are left at once; and one resident wave of
// blocks keeps the occupancy words instead of loading them for every 8 queries.
// 65 536 queries of a sheet on itself 80.5 -> 63 us, on a sphere 26 -> 18,
// 4096 on a box of 12 faces 14.7 -> 10.1; 6 blocks an SM (4: 70 us, 8: 62 but 25
// on the sphere).
constexpr int CT_BLOCK = 256;
constexpr int CT_LONG_CELL = 20;

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += o;
    }
    return v;
}
// lowest lane whose inclusive count exceeds k (31 when none does)
__device__ __forceinline__ int warp_owner(int incl, int k) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1)
        if (__shfl_sync(0xffffffffu, incl, lo + step - 1) <= k) lo += step;
    return lo;
}

// EDGE: query q is the box of edge q (endpoints edges[2q], edges[2q+1] in p4)
// grown by pad (XPBD.py:221-232), else the box p4[q] +- pad.
template <bool EDGE>
__global__ void __launch_bounds__(CT_BLOCK, 6) cell_traverse_kernel(
    int Q, const float4* __restrict__ p4, float pad, const float* __restrict__ grid8, const float* __restrict__ box6,
    const float4* __restrict__ nmin4, const float4* __restrict__ nmax4, const int* __restrict__ prefix,
    const float4* __restrict__ frec, int cap, int* __restrict__ cand, int* __restrict__ num, int* status,
    const int* __restrict__ edges) {
    pdl_entry();
    // occupancy words: bit z of word x*32 + y = cell (x, y, z) holds faces
    __shared__ unsigned occ[kGridRes * kGridRes];
    const unsigned* gocc = reinterpret_cast<const unsigned*>(grid8) + kGridHeader;
    for (int k = threadIdx.x; k < kGridRes * kGridRes; k += blockDim.x) occ[k] = gocc[k];
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    const unsigned below = (1u << lane) - 1u;
    // lanes 0, 1, 2 (and all further ones, as 2): this lane's axis
    const int axis = min(lane, 2);
    const float cell = grid8[axis], reach = grid8[3 + axis], origin = box6[axis];
    const float* p = reinterpret_cast<const float*>(p4) + axis;
    for (int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < Q; q += nw) {  // warp-uniform
        float qa, qb;
        if (EDGE) {
            const float p0 = p[4 * (size_t)edges[2 * q]], p1 = p[4 * (size_t)edges[2 * q + 1]];
            qa = fminf(p0, p1) - pad;
            qb = fmaxf(p0, p1) + pad;
        } else {
            const float p0 = p[4 * (size_t)q];
            qa = p0 - pad;
            qb = p0 + pad;
        }
        const int ic = f2i_sat((0.5f * (qa + qb) - origin) / cell);
        int i0, i1;
        cell_range(qa, qb, origin, cell, reach, &i0, &i1);
        const int ix = __shfl_sync(0xffffffffu, ic, 0), iy = __shfl_sync(0xffffffffu, ic, 1),
                  iz = __shfl_sync(0xffffffffu, ic, 2);
        const V3 a{__shfl_sync(0xffffffffu, qa, 0), __shfl_sync(0xffffffffu, qa, 1), __shfl_sync(0xffffffffu, qa, 2)};
        const V3 b{__shfl_sync(0xffffffffu, qb, 0), __shfl_sync(0xffffffffu, qb, 1), __shfl_sync(0xffffffffu, qb, 2)};
        const int cid =
            (int)((unsigned)ix * (unsigned)(kGridRes * kGridRes) + (unsigned)iy * (unsigned)kGridRes + (unsigned)iz);
        int count = 0;  // warp-uniform
        int* out = cand + (size_t)q * cap;
        if (cid <= kNumCells - 1) {  // the reference's skip rule (lbvh_cell.py:665)
            const int x0 = __shfl_sync(0xffffffffu, i0, 0), x1 = __shfl_sync(0xffffffffu, i1, 0);
            const int y0 = __shfl_sync(0xffffffffu, i0, 1), y1 = __shfl_sync(0xffffffffu, i1, 1);
            const int z0 = __shfl_sync(0xffffffffu, i0, 2), z1 = __shfl_sync(0xffffffffu, i1, 2);
            if (z0 <= z1 && x0 <= x1 && y0 <= y1) {
                const unsigned zmask = (z1 == 31 ? 0xffffffffu : ((1u << (z1 + 1)) - 1u)) & ~((1u << z0) - 1u);
                const int ny = y1 - y0 + 1, ncol = (x1 - x0 + 1) * ny;
                // columns in visiting order (x descending, then y descending), 32 at a time
                for (int c0 = 0; c0 < ncol; c0 += 32) {
                    unsigned cm = 0u;  // this lane's column: occupied cells within the z range
                    if (c0 + lane < ncol) {
                        const int cc = c0 + lane;
                        cm = occ[(x1 - cc / ny) * kGridRes + (y1 - cc % ny)] & zmask;
                    }
                    if (!__any_sync(0xffffffffu, cm != 0u)) continue;
                    const int cn = __popc(cm);
                    const int cincl = warp_incl_scan(cn, lane);
                    const int ctotal = __shfl_sync(0xffffffffu, cincl, 31);
                    // the occupied cells of these columns end to end (z descending
                    // within a column), 32 at a time: lane k takes the k-th
                    for (int k0 = 0; k0 < ctotal; k0 += 32) {
                        const int k = k0 + lane;
                        const int oc = warp_owner(cincl, k);
                        const unsigned m = __shfl_sync(0xffffffffu, cm, oc);
                        const int rank = k - (__shfl_sync(0xffffffffu, cincl, oc) - __shfl_sync(0xffffffffu, cn, oc));
                        int start = 0, n = 0;
                        if (k < ctotal) {
                            // position of the rank-th highest set bit of m
                            int cz = 0;
    #pragma unroll
                            for (int step = 16; step >= 1; step >>= 1)
                                if (__popc(m >> (cz + step)) >= rank + 1) cz += step;
                            const int cc = c0 + oc;
                            const int i = (x1 - cc / ny) * kGridRes * kGridRes + (y1 - cc % ny) * kGridRes + cz;
                            const int leaf = i + kNumCells - 1;
                            if (overlap(a, b, mk(nmin4[leaf]), mk(nmax4[leaf]))) {
                                start = i == 0 ? 0 : prefix[i - 1];
                                n = prefix[i] - start;
                            }
                        }
                        unsigned full = __ballot_sync(0xffffffffu, n > 0);
                        const int total = __reduce_add_sync(0xffffffffu, n);
                        if (total >= CT_LONG_CELL * __popc(full)) {
                            // long cells: one after the other
                            for (; full != 0u; full &= full - 1u) {
                                const int l = __ffs(full) - 1;
                                const int o_start = __shfl_sync(0xffffffffu, start, l);
                                const int o_n = __shfl_sync(0xffffffffu, n, l);
                                for (int f0 = 0; f0 < o_n; f0 += 32) {
                                    bool hit = false;
                                    float4 fa = make_float4(0.f, 0.f, 0.f, 0.f);
                                    if (f0 + lane < o_n) {
                                        fa = frec[2 * (o_start + f0 + lane)];
                                        hit = overlap(a, b, mk(fa), mk(frec[2 * (o_start + f0 + lane) + 1]));
                                    }
                                    const unsigned hits = __ballot_sync(0xffffffffu, hit);
                                    if (hit) {
                                        const int slot = count + __popc(hits & below);
                                        if (slot < cap) out[slot] = __float_as_int(fa.w);
                                    }
                                    count += __popc(hits);
                                }
                            }
                            continue;
                        }
                        const int incl = warp_incl_scan(n, lane);  // faces of the passing cells, in order
                        for (int f0 = 0; f0 < total; f0 += 32) {
                            const int f = f0 + lane;
                            const int lo = warp_owner(incl, f);
                            const int o_incl = __shfl_sync(0xffffffffu, incl, lo);
                            const int o_n = __shfl_sync(0xffffffffu, n, lo);
                            const int o_start = __shfl_sync(0xffffffffu, start, lo);
                            bool hit = false;
                            float4 fa = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (f < total) {
                                const int j = o_start + (f - (o_incl - o_n));
                                fa = frec[2 * j];
                                hit = overlap(a, b, mk(fa), mk(frec[2 * j + 1]));
                            }
                            const unsigned hits = __ballot_sync(0xffffffffu, hit);
                            if (hit) {
                                const int slot = count + __popc(hits & below);
                                if (slot < cap) out[slot] = __float_as_int(fa.w);
                            }
                            count += __popc(hits);
                        }
                    }
                }
            }
        }
        if (lane == 0) {
            num[q] = count;
            if (count > cap) atomicOr(status, SX_STATUS_CAND_OVERFLOW);
        }
    }
}

// ---------------------------------------------------------------------------
// Face-level LBVH refit and traversal
// ---------------------------------------------------------------------------
__global__ void face_refit_kernel(int n, const int* __restrict__ sorted_ids, const float4* __restrict__ fmn4,
                                  const float4* __restrict__ fmx4, const int* __restrict__ child_a,
                                  const int* __restrict__ child_b, const int* __restrict__ parent, float4* nmin4,
                                  float4* nmax4, int* flags, int* status) {
    pdl_entry();
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int leaf = n - 1 + j, f = sorted_ids[j];
    nmin4[leaf] = fmn4[f];
    nmax4[leaf] = fmx4[f];
    if (n == 1) return;
    int node = parent[leaf];
    for (int steps = 0; node >= 0; ++steps) {
        if (steps > n) {
            atomicOr(status, SX_STATUS_CLIMB_LIMIT);
            return;
        }
        __threadfence();
        if (atomicAdd(flags + node, 1) == 0) return;
        flags[node] = 0;
        const int l = child_a[node], r = child_b[node];
        V3 a = vmin(load_cg(nmin4 + l), load_cg(nmin4 + r));
        V3 b = vmax(load_cg(nmax4 + l), load_cg(nmax4 + r));
        store_box(nmin4, nmax4, node, a, b);
        node = parent[node];
    }
}

// The same refit with its lower levels in shared memory.  A Karras node
// covers a contiguous range of sorted leaves and carries the index of one of
// its ends, so every node whose range lies inside a block's tile of 256 leaves
// has its index in the tile as well: the block keeps those nodes' boxes and
// arrival counters in shared memory (block-scope fences, no global atomics).
// A thread that climbs out of the tile continues with the global protocol of
// face_refit_kernel.  Each thread carries its current box in registers; every
// internal box is also written to global memory.  Min and max are exact, so
// the boxes are the same as the one-thread-per-leaf climb's.
constexpr int FR_TILE = 256;

// node c (internal 0..n-2 or leaf n-1+j) has its slot in the tile [B, tile_end]
__device__ __forceinline__ bool in_tile(int c, int n, int B, int tile_end) {
    const int k = c >= n - 1 ? c - (n - 1) : c;
    return k >= B && k <= tile_end;
}

__global__ void __launch_bounds__(FR_TILE) face_refit_tiled_kernel(
    int n, const int* __restrict__ sorted_ids, const float4* __restrict__ fmn4, const float4* __restrict__ fmx4,
    const int* __restrict__ child_a, const int* __restrict__ child_b, const int* __restrict__ parent,
    const int* __restrict__ range_l, const int* __restrict__ range_r, float4* nmin4, float4* nmax4, int* flags,
    int* status) {
    pdl_entry();
    __shared__ float4 s_leaf[2][FR_TILE];
    __shared__ float4 s_node[2][FR_TILE];
    __shared__ int s_flag[FR_TILE];
    const int B = blockIdx.x * FR_TILE, t = threadIdx.x, j = B + t;
    s_flag[t] = 0;
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (j < n) {
        const int f = sorted_ids[j];
        lo = fmn4[f];
        hi = fmx4[f];
        nmin4[n - 1 + j] = lo;
        nmax4[n - 1 + j] = hi;
        s_leaf[0][t] = lo;
        s_leaf[1][t] = hi;
    }
    __syncthreads();
    if (j >= n || n == 1) return;
    const int tile_end = min(B + FR_TILE, n) - 1;  // last leaf of the tile
    int me = n - 1 + j;
    int node = parent[me];
    bool local = true;
    // topology of the current node; the next level's is loaded before this
    // level's arrival counter, so that only the counter and the sibling's box
    // are round trips on the climb's critical path
    int ca = 0, cb = 0, up = -1, rl = 0, rr = 0;
    if (node >= 0) {
        ca = __ldg(child_a + node); cb = __ldg(child_b + node); up = __ldg(parent + node);
        rl = __ldg(range_l + node); rr = __ldg(range_r + node);
    }
    for (int steps = 0; node >= 0; ++steps) {
        if (steps > n) {
            atomicOr(status, SX_STATUS_CLIMB_LIMIT);
            return;
        }
        int nca = 0, ncb = 0, nup = -1, nrl = 0, nrr = 0;
        if (up >= 0) {
            nca = __ldg(child_a + up); ncb = __ldg(child_b + up); nup = __ldg(parent + up);
            nrl = __ldg(range_l + up); nrr = __ldg(range_r + up);
        }
        const int sib = ca == me ? cb : ca;
        float4 slo, shi;
        // local: the node and both children lie in the tile (decided from the
        // node alone, so both children agree; always true below a node whose
        // range is in the tile when the hierarchy is well formed)
        if (local && node >= B && node <= tile_end && rl >= B && rr <= tile_end && in_tile(ca, n, B, tile_end) &&
            in_tile(cb, n, B, tile_end)) {
            __threadfence_block();
            if (atomicAdd(s_flag + (node - B), 1) == 0) return;
            __threadfence_block();
            const bool sib_leaf = sib >= n - 1;
            const int k = sib_leaf ? sib - (n - 1) - B : sib - B;
            slo = sib_leaf ? s_leaf[0][k] : s_node[0][k];
            shi = sib_leaf ? s_leaf[1][k] : s_node[1][k];
        } else {
            local = false;
            // release: this thread's box stores are visible before the count;
            // acquire: the sibling's are visible to the loads below
            cuda::atomic_ref<int, cuda::thread_scope_device> cnt(flags[node]);
            if (cnt.fetch_add(1, cuda::memory_order_acq_rel) == 0) return;
            flags[node] = 0;
            slo = __ldcg(nmin4 + sib);
            shi = __ldcg(nmax4 + sib);
        }
        const V3 a = vmin(mk(lo), mk(slo)), b = vmax(mk(hi), mk(shi));
        store_box(nmin4, nmax4, node, a, b);
        lo = make_float4(a.x, a.y, a.z, 0.f);
        hi = make_float4(b.x, b.y, b.z, 0.f);
        if (local) {
            s_node[0][node - B] = lo;
            s_node[1][node - B] = hi;
        }
        me = node;
        node = up;
        ca = nca; cb = ncb; up = nup; rl = nrl; rr = nrr;
    }
}

// ---------------------------------------------------------------------------
// Refit by ranges, and child records for the queries.
//
// Entry e of level k >= 1 is the union of the sorted leaves 8^k e .. 8^k (e + 1)
// - 1, {min, max} in 32 bytes; a level is padded with empty boxes to whole
// groups of 8 and the last one is a single group.  A Karras node covers a
// contiguous range of leaves, so its box is the union of at most 7 + 7 entries
// per level: no climb, whose last 20-25 levels are two dependent round trips
// each (101 us for 2^20 leaves, without the records below; this takes 81, for
// 20 011 leaves 27 -> 11).  Min and max are exact, so the boxes are the
// climb's bit for bit.
//
// Record i holds both children of internal node i, {min, id}, {max, -} each, the
// id an internal node's index or ~face: a query reads one line per node in one
// round trip instead of the two child indices and then four boxes from four
// places.  Every node writes its own half of its parent's record.
// ---------------------------------------------------------------------------
constexpr int LV_MAX = 12;  // 8^11 > 2^31
struct LevelTable {
    int top;               // level of the single group
    long long off[LV_MAX]; // first entry of level k >= 1
    int count[LV_MAX];     // entries of level k without padding
};
static LevelTable level_table(int n) {
    LevelTable t = {};
    t.count[0] = n;
    long long at = 0;
    int k = 0;
    while (t.count[k] > 8) {
        t.count[k + 1] = (int)((t.count[k] + 7LL) / 8);
        t.off[k + 1] = at;
        at += (t.count[k + 1] + 7LL) / 8 * 8;
        ++k;
    }
    t.top = k;
    return t;
}
static long long level_entries(int n) {
    const LevelTable t = level_table(n);
    return t.top == 0 ? 0 : t.off[t.top] + 8;
}
__device__ __forceinline__ void put_child(float4* rec, int parent, bool right, V3 a, V3 b, int id) {
    float4* r = rec + 4 * (size_t)parent + (right ? 2 : 0);
    r[0] = make_float4(a.x, a.y, a.z, __int_as_float(id));
    r[1] = make_float4(b.x, b.y, b.z, 0.0f);
}

__device__ __forceinline__ void join_lanes(V3& a, V3& b, int width) {
    for (int o = 1; o < width; o <<= 1) {
        a = vmin(a, V3{__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                       __shfl_xor_sync(0xffffffffu, a.z, o)});
        b = vmax(b, V3{__shfl_xor_sync(0xffffffffu, b.x, o), __shfl_xor_sync(0xffffffffu, b.y, o),
                       __shfl_xor_sync(0xffffffffu, b.z, o)});
    }
}
__device__ __forceinline__ void put_entry(float4* lv, long long e, V3 a, V3 b) {
    lv[2 * e] = make_float4(a.x, a.y, a.z, 0.0f);
    lv[2 * e + 1] = make_float4(b.x, b.y, b.z, 0.0f);
}

// Leaf boxes in sorted order and levels 1 and 2 (a block covers 256 leaves: 32
// entries of level 1, 4 of level 2).
__device__ __forceinline__ void join_box(V3& a, V3& b, float4 lo, float4 hi) {
    a = vmin(a, mk(lo));
    b = vmax(b, mk(hi));
}
__global__ void __launch_bounds__(256) face_leaves_kernel(int n, const int* __restrict__ sorted_ids,
                                                          const float4* __restrict__ fmn4,
                                                          const float4* __restrict__ fmx4,
                                                          const int* __restrict__ parent,
                                                          const int* __restrict__ range_l,
                                                          float4* __restrict__ nmin4, float4* __restrict__ nmax4,
                                                          float4* __restrict__ lv, float4* __restrict__ rec,
                                                          LevelTable t) {
    pdl_entry();
    const int j = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31;
    V3 a{INFINITY, INFINITY, INFINITY}, b{-INFINITY, -INFINITY, -INFINITY};
    if (j < n) {
        const int f = sorted_ids[j];
        const float4 lo = fmn4[f], hi = fmx4[f];
        nmin4[n - 1 + j] = lo;
        nmax4[n - 1 + j] = hi;
        a = mk(lo);
        b = mk(hi);
        if (n > 1) {
            const int p = parent[n - 1 + j];
            put_child(rec, p, range_l[p] != j, a, b, ~f);
        }
    }
    if (t.top < 1) return;
    join_lanes(a, b, 8);
    const int e1 = j >> 3;
    const bool own = (lane & 7) == 0;
    if (own && e1 < (t.count[1] + 7) / 8 * 8) put_entry(lv, t.off[1] + e1, a, b);
    if (t.top < 2) return;
    __shared__ V3 sa[32], sb[32];
    if (own) {
        sa[threadIdx.x >> 3] = a;
        sb[threadIdx.x >> 3] = b;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        a = sa[threadIdx.x];
        b = sb[threadIdx.x];
        join_lanes(a, b, 8);
        const int e2 = blockIdx.x * 4 + (lane >> 3);
        if (own && e2 < (t.count[2] + 7) / 8 * 8) put_entry(lv, t.off[2] + e2, a, b);
    }
}

// Level k from level k - 1, 8 lanes per entry, padding included; the last
// blocks' padding of level k - 1 holds empty boxes already.
__global__ void __launch_bounds__(256) face_level_kernel(float4* lv, LevelTable t, int k) {
    pdl_entry();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x, e = i >> 3;
    const long long padded = (t.count[k] + 7) / 8 * 8;
    V3 a{INFINITY, INFINITY, INFINITY}, b{-INFINITY, -INFINITY, -INFINITY};
    if (i < t.count[k - 1]) {
        a = mk(lv[2 * (t.off[k - 1] + i)]);
        b = mk(lv[2 * (t.off[k - 1] + i) + 1]);
    }
    join_lanes(a, b, 8);
    if ((threadIdx.x & 7) == 0 && e < padded) put_entry(lv, t.off[k] + e, a, b);
}

// Levels k0 .. top in one block.
__global__ void __launch_bounds__(1024) face_top_levels_kernel(float4* lv, LevelTable t, int k0) {
    pdl_entry();
    for (int k = k0; k <= t.top; ++k) {
        const int padded = (t.count[k] + 7) / 8 * 8;
        for (int i0 = 0; i0 < 8 * padded; i0 += 1024) {
            const int i = i0 + threadIdx.x;
            V3 a{INFINITY, INFINITY, INFINITY}, b{-INFINITY, -INFINITY, -INFINITY};
            if (i < t.count[k - 1]) {
                a = mk(lv[2 * (t.off[k - 1] + i)]);
                b = mk(lv[2 * (t.off[k - 1] + i) + 1]);
            }
            join_lanes(a, b, 8);
            if ((threadIdx.x & 7) == 0 && i < 8 * padded) put_entry(lv, t.off[k] + (i >> 3), a, b);
        }
        __syncthreads();
    }
}

// Internal node i: the union over its range of leaves.  (Nodes inside a block's
// 256 leaves taken from shared memory in the leaf kernel instead: 88 against 81
// us for the whole refit of 2^20 leaves.)
__global__ void __launch_bounds__(256) face_ranges_kernel(int n, const int* __restrict__ range_l,
                                                          const int* __restrict__ range_r,
                                                          const int* __restrict__ parent, float4* nmin4,
                                                          float4* nmax4, const float4* __restrict__ lv,
                                                          float4* __restrict__ rec, LevelTable t) {
    pdl_entry();
    __shared__ long long off[LV_MAX];
    if (threadIdx.x < LV_MAX) off[threadIdx.x] = t.off[threadIdx.x];
    __syncthreads();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n - 1) return;
    const int l = range_l[i], r = range_r[i];
    V3 a{NAN, NAN, NAN}, b{NAN, NAN, NAN};  // fminf and fmaxf pass over a NaN
    int lo = l, hi = r + 1;  // [lo, hi)
    const float4 *mn = nmin4 + (n - 1), *mx = nmax4 + (n - 1);
    int step = 1;
    for (int k = 0;; ++k) {
        const int l1 = k == t.top ? hi : min((lo + 7) & ~7, hi), h0 = max(hi & ~7, l1);
        for (int e = lo; e < l1; ++e) join_box(a, b, mn[(size_t)e * step], mx[(size_t)e * step]);
        for (int e = h0; e < hi; ++e) join_box(a, b, mn[(size_t)e * step], mx[(size_t)e * step]);
        if (l1 >= h0) break;
        lo = l1 >> 3;
        hi = h0 >> 3;
        mn = lv + 2 * off[k + 1];
        mx = mn + 1;
        step = 2;
    }
    store_box(nmin4, nmax4, i, a, b);
    if (i > 0) put_child(rec, parent[i], l == i, a, b, i);  // a right child carries its first leaf's index
}

// face_traverse_kernel over the child records: the same visiting order (right
// child first), so the same candidates in the same order.  A leaf that is next
// in that order is reported where its parent is tested, without a push and a pop.
__global__ void __launch_bounds__(128) face_query_kernel(int n, int Q, const float4* __restrict__ p4, float pad,
                                                         const int* __restrict__ sorted_ids,
                                                         const float4* __restrict__ nmin4,
                                                         const float4* __restrict__ nmax4,
                                                         const float4* __restrict__ rec, int cap,
                                                         int* __restrict__ cand, int* __restrict__ num, int* status,
                                                         const int* __restrict__ order) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Q) return;
    const int q = order ? order[i] : i;
    const V3 p = mk(p4[q]);
    const V3 a{p.x - pad, p.y - pad, p.z - pad}, b{p.x + pad, p.y + pad, p.z + pad};
    int count = 0, flags = 0;
    int* out = cand + (size_t)q * cap;
    auto report = [&](int face) {
        if (count < cap) out[count] = face;
        ++count;
    };
    int stack[64];
    int sc = 0;
    if (n == 1) {
        if (overlap(a, b, mk(nmin4[0]), mk(nmax4[0]))) report(sorted_ids[0]);
    } else {
        int cur = 0;
        for (long long visits = 0;; ++visits) {
            if (visits > 2LL * n) {  // each node is visited at most once
                flags |= SX_STATUS_STACK_OVERFLOW;
                break;
            }
            const float4* r4 = rec + 4 * (size_t)cur;
            const float4 la = r4[0], lb = r4[1], ra = r4[2], rb = r4[3];
            bool hl = overlap(a, b, mk(la), mk(lb)), hr = overlap(a, b, mk(ra), mk(rb));
            const int l = __float_as_int(la.w), r = __float_as_int(ra.w);
            if (hr && r < 0) {
                report(~r);
                hr = false;
            }
            if (hl && l < 0 && !hr) {
                report(~l);
                hl = false;
            }
            if (hr) {
                if (hl) {
                    if (sc < 64) stack[sc++] = l; else flags |= SX_STATUS_STACK_OVERFLOW;
                }
                cur = r;
            } else if (hl) {
                cur = l;
            } else {
                cur = -1;
                while (sc > 0) {
                    cur = stack[--sc];
                    if (cur >= 0) break;
                    report(~cur);
                }
                if (cur < 0) break;
            }
        }
    }
    num[q] = count;
    if (count > cap) flags |= SX_STATUS_CAND_OVERFLOW;
    if (flags) atomicOr(status, flags);
}

__global__ void __launch_bounds__(128) face_traverse_kernel(int n, int Q, const float4* __restrict__ p4, float pad,
                                                            const int* __restrict__ child_a,
                                                            const int* __restrict__ child_b,
                                                            const int* __restrict__ sorted_ids,
                                                            const float4* __restrict__ nmin4,
                                                            const float4* __restrict__ nmax4, int cap,
                                                            int* __restrict__ cand, int* __restrict__ num,
                                                            int* status, const int* __restrict__ order) {
    pdl_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Q) return;
    // order (optional): the queries in a spatially coherent order, so that a
    // warp's threads walk nearby parts of the tree
    const int q = order ? order[i] : i;
    V3 p = mk(p4[q]);
    V3 a{p.x - pad, p.y - pad, p.z - pad}, b{p.x + pad, p.y + pad, p.z + pad};
    int count = 0, flags = 0;
    int* out = cand + (size_t)q * cap;
    int stack[64];
    int sc = 0;
    // Children are tested before they are pushed (same visiting order as a
    // pop-time test, see cell_traverse_kernel).
    if (overlap(a, b, mk(nmin4[0]), mk(nmax4[0]))) stack[sc++] = 0;
    // A well-formed tree pops each of its 2n-1 nodes at most once; the bound
    // stops the walk on a malformed hierarchy (reference tie rule with repeated
    // codes can create cycles).
    long long pops = 0;
    const long long max_pops = 2LL * n;
    while (sc > 0) {
        if (++pops > max_pops) {
            flags |= SX_STATUS_STACK_OVERFLOW;
            break;
        }
        const int idx = stack[--sc];
        if (idx >= n - 1) {
            if (count < cap) out[count] = sorted_ids[idx - (n - 1)];
            ++count;
        } else {
            const int l = child_a[idx], r = child_b[idx];
            if (overlap(a, b, mk(nmin4[l]), mk(nmax4[l]))) {
                if (sc < 64) stack[sc++] = l; else flags |= SX_STATUS_STACK_OVERFLOW;
            }
            if (overlap(a, b, mk(nmin4[r]), mk(nmax4[r]))) {
                if (sc < 64) stack[sc++] = r; else flags |= SX_STATUS_STACK_OVERFLOW;
            }
        }
    }
    num[q] = count;
    if (count > cap) flags |= SX_STATUS_CAND_OVERFLOW;
    if (flags) atomicOr(status, flags);
}

}  // namespace sx

using namespace sx;

// ---- workspace layouts --------------------------------------------------------
// cell BVH: [keys F][radix ws F] ; init uses [codes NC][radix ws NC]
extern "C" size_t sx_radix_sort_workspace_bytes(int n) { return rs_ws_bytes(n); }

extern "C" size_t sx_cell_bvh_workspace_bytes(int n_faces) {
    size_t build = align256((size_t)(n_faces > 0 ? n_faces : 1) * 4) + rs_ws_bytes(n_faces) +
                   align256((size_t)kNumCells * 4);
    size_t init = align256((size_t)kNumCells * 4) + rs_ws_bytes(kNumCells);
    return build > init ? build : init;
}

extern "C" int sx_radix_sort_pairs(unsigned* keys, int* vals, int n, int bits, void* ws, size_t ws_bytes,
                                   void* stream) {
    SX_REQUIRE(n >= 0, "sx_radix_sort_pairs: n < 0");
    if (n <= 1) return SX_OK;
    SX_REQUIRE(keys && vals, "sx_radix_sort_pairs: null pointer");
    return radix_sort(keys, vals, n, bits, ws, ws_bytes, as_stream(stream));
}

extern "C" int sx_radix_sort_pairs_bits(unsigned* keys, int* vals, int n, int first_bit, int bits, void* ws,
                                        size_t ws_bytes, void* stream) {
    SX_REQUIRE(n >= 0, "sx_radix_sort_pairs_bits: n < 0");
    if (n <= 1) return SX_OK;
    SX_REQUIRE(keys && vals, "sx_radix_sort_pairs_bits: null pointer");
    return radix_sort(keys, vals, n, bits, ws, ws_bytes, as_stream(stream), first_bit);
}

// ---------------------------------------------------------------------------
// Radix sort without a caller-provided workspace.
//
// Some callers cannot allocate device memory when they need to sort: hosts
// whose device memory belongs to another allocator with a fixed budget (a
// framework's caching pool, an engine's arena), where an extra cudaMalloc can
// fail or fragment the pool, and real-time loops that cannot afford the
// device-wide synchronisation cudaMalloc/cudaFree may cause.  For them the
// sort's scratch (two key/value ping-pong buffers and the digit histograms)
// lives in one fixed array in this library's device memory, sized for at most
// kNoAllocMaxKeys keys.  Every GPU that loads the library keeps the array
// (about 2.1 MB) until the process exits.
//
// In host code the array's name is only a host-side stand-in for the symbol, so
// its device address is looked up once per device, on the first call made with
// that device current, with cudaGetSymbolAddress; that first call should come
// before any stream capture.  The cached address is never refreshed: a
// cudaDeviceReset re-creates the context and may move the array, so callers
// must not use this entry point after resetting the device.  All calls share the array: calls that overlap on
// the GPU (different streams, or threads) race on it and must be ordered by the
// caller.  Nothing in it needs clearing: every pass overwrites the histogram
// and both ping-pong buffers before reading them.
// ---------------------------------------------------------------------------
constexpr int kNoAllocMaxKeys = 1 << 18;
constexpr size_t kNoAllocScratchBytes =
    2 * (((size_t)kNoAllocMaxKeys * 4 + 255) & ~(size_t)255) +
    (((size_t)256 * ((kNoAllocMaxKeys + RS_TILE - 1) / RS_TILE) * 4 + 255) & ~(size_t)255) + 256 * 4;
static __device__ __align__(256) unsigned char g_sort_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
static std::mutex g_scratch_mutex;
static void* g_scratch_addr[kMaxDevices] = {};

static int sort_scratch_for_current_device(void** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
    SX_REQUIRE(dev >= 0 && dev < kMaxDevices, "sx_radix_sort_pairs_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_sort_scratch);
        if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(g_sort_scratch)");
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return SX_OK;
}

extern "C" int sx_radix_sort_pairs_noalloc(unsigned* keys, int* vals, int n, int bits, void* stream) {
    SX_REQUIRE(n >= 0, "sx_radix_sort_pairs_noalloc: n < 0");
    SX_REQUIRE(n <= kNoAllocMaxKeys,
               "sx_radix_sort_pairs_noalloc: %d keys exceed the fixed scratch capacity of %d keys; "
               "use sx_radix_sort_pairs with a workspace",
               n, kNoAllocMaxKeys);
    if (n <= 1) return SX_OK;
    SX_REQUIRE(keys && vals, "sx_radix_sort_pairs_noalloc: null pointer");
    SX_REQUIRE(rs_ws_bytes(n) <= kNoAllocScratchBytes, "sx_radix_sort_pairs_noalloc: scratch layout mismatch");
    void* scratch = nullptr;
    int rc = sort_scratch_for_current_device(&scratch);
    if (rc) return rc;
    return radix_sort(keys, vals, n, bits, scratch, kNoAllocScratchBytes, as_stream(stream));
}

extern "C" int sx_face_morton(const float* fmin4, const float* fmax4, int n_faces, const float* box6,
                              unsigned* codes, int* ids, void* stream) {
    SX_REQUIRE(n_faces >= 0, "sx_face_morton: n_faces < 0");
    if (n_faces == 0) return SX_OK;
    SX_REQUIRE(fmin4 && fmax4 && box6 && codes && ids, "sx_face_morton: null pointer");
    launch(face_morton_kernel, grid_for(n_faces, 256), 256, 0, as_stream(stream), 
        n_faces, (const float4*)fmin4, (const float4*)fmax4, box6, codes, ids);
    return check_launch("face_morton_kernel");
}

extern "C" int sx_karras_build(const unsigned* codes, int n, int tie, int* child_a, int* child_b, int* range_l,
                               int* range_r, int* parent, void* stream) {
    SX_REQUIRE(n >= 1, "sx_karras_build: n must be >= 1");
    SX_REQUIRE(codes && parent && (n == 1 || (child_a && child_b && range_l && range_r)),
               "sx_karras_build: null pointer");
    launch(karras_kernel, grid_for(n, 256), 256, 0, as_stream(stream), n, codes, tie ? 1 : 0, child_a, child_b,
                                                                    range_l, range_r, parent);
    return check_launch("karras_kernel");
}

extern "C" int sx_cell_bvh_init(int* sorted_codes, int* sorted_ids, int* child_a, int* child_b, int* range_l,
                                int* range_r, int* parent, void* ws, size_t ws_bytes, void* stream) {
    SX_REQUIRE(sorted_codes && sorted_ids && child_a && child_b && range_l && range_r && parent,
               "sx_cell_bvh_init: null pointer");
    SX_REQUIRE(ws && ws_bytes >= sx_cell_bvh_workspace_bytes(0), "sx_cell_bvh_init: workspace too small");
    cudaStream_t s = as_stream(stream);
    launch(cell_morton_kernel, grid_for(kNumCells, 256), 256, 0, s, (unsigned*)sorted_codes, sorted_ids);
    int rc = check_launch("cell_morton_kernel");
    if (rc) return rc;
    rc = radix_sort((unsigned*)sorted_codes, sorted_ids, kNumCells, 30, ws, ws_bytes, s);
    if (rc) return rc;
    launch(karras_kernel, grid_for(kNumCells, 256), 256, 0, s, kNumCells, (const unsigned*)sorted_codes, 0, child_a,
                                                           child_b, range_l, range_r, parent);
    return check_launch("karras_kernel(cells)");
}

extern "C" int sx_cell_bvh_build_copy(const float* fmin4, const float* fmax4, int n_faces, const float* box6,
                                      float* box_out6, const int* child_a, const int* child_b, const int* parent,
                                      int* sorted_face_ids, int* prefix, int* num_faces, float* nmin4, float* nmax4,
                                      float* face_rec8, float* grid8, void* ws, size_t ws_bytes, void* stream) {
    SX_REQUIRE(n_faces >= 0, "sx_cell_bvh_build: n_faces < 0");
    SX_REQUIRE(box6 && child_a && child_b && parent && prefix && num_faces && nmin4 && nmax4 && grid8,
               "sx_cell_bvh_build: null pointer");
    SX_REQUIRE(n_faces == 0 || (fmin4 && fmax4 && sorted_face_ids && face_rec8),
               "sx_cell_bvh_build: null face arrays");
    SX_REQUIRE(ws && ws_bytes >= sx_cell_bvh_workspace_bytes(n_faces), "sx_cell_bvh_build: workspace too small");
    cudaStream_t s = as_stream(stream);
    char* p = (char*)ws;
    unsigned* keys = (unsigned*)p;
    p += align256((size_t)(n_faces > 0 ? n_faces : 1) * 4);
    void* rws = p;
    launch(face_cell_kernel, grid_for(n_faces > 0 ? n_faces : 1, 256), 256, 0, s, n_faces, (const float4*)fmin4,
           (const float4*)fmax4, box6, box_out6, keys, sorted_face_ids, grid8);
    int rc = check_launch("face_cell_kernel");
    if (rc) return rc;
    if (n_faces > 1) {
        rc = radix_sort(keys, sorted_face_ids, n_faces, 15, rws, rs_ws_bytes(n_faces), s);
        if (rc) return rc;
    }
    launch(cell_bounds_kernel, grid_for((long long)n_faces + 1, 256), 256, 0, s, n_faces, (const unsigned*)keys, prefix);
    launch(cell_column_refit_kernel, kGridRes * kGridRes, kColumnRefitThreads, 0, s, box6, (const int*)prefix,
           (const int*)sorted_face_ids, (const float4*)fmin4, (const float4*)fmax4, num_faces, (float4*)nmin4,
           (float4*)nmax4, (float4*)face_rec8, grid8);
    return check_launch("cell_column_refit_kernel");
}

extern "C" int sx_cell_bvh_build(const float* fmin4, const float* fmax4, int n_faces, const float* box6,
                                 const int* child_a, const int* child_b, const int* parent, int* sorted_face_ids,
                                 int* prefix, int* num_faces, float* nmin4, float* nmax4, float* face_rec8,
                                 float* grid8, void* ws, size_t ws_bytes, void* stream) {
    return sx_cell_bvh_build_copy(fmin4, fmax4, n_faces, box6, nullptr, child_a, child_b, parent, sorted_face_ids,
                                  prefix, num_faces, nmin4, nmax4, face_rec8, grid8, ws, ws_bytes, stream);
}

// a warp a query, at most one resident wave of blocks
template <typename K>
static int traverse_grid(K kernel, int queries) {
    const int g = grid_for(32LL * queries, CT_BLOCK), cap = resident_blocks(kernel, CT_BLOCK);
    return g < cap ? g : cap;
}

extern "C" int sx_cell_bvh_traverse(const float* p4, int n_queries, float padding, const float* grid8,
                                    const float* origin_box6, const float* nmin4, const float* nmax4,
                                    const int* prefix,
                                    const float* face_rec8, int cap, int* cand, int* num, int* status,
                                    void* stream) {
    SX_REQUIRE(n_queries >= 0 && cap >= 1, "sx_cell_bvh_traverse: bad sizes");
    if (n_queries == 0) return SX_OK;
    SX_REQUIRE(p4 && grid8 && origin_box6 && nmin4 && nmax4 && prefix && face_rec8 &&
                   cand && num && status,
               "sx_cell_bvh_traverse: null pointer");
    launch(cell_traverse_kernel<false>, traverse_grid(cell_traverse_kernel<false>, n_queries), CT_BLOCK, 0,
           as_stream(stream), n_queries, (const float4*)p4, padding, grid8, origin_box6, (const float4*)nmin4,
           (const float4*)nmax4, prefix, (const float4*)face_rec8, cap, cand, num, status, (const int*)nullptr);
    return check_launch("cell_traverse_kernel");
}

extern "C" int sx_cell_bvh_traverse_edges(const int* edges, int n_edges, const float* p4, float padding,
                                          const float* grid8, const float* origin_box6, const float* nmin4,
                                          const float* nmax4, const int* prefix, const float* face_rec8, int cap,
                                          int* cand, int* num, int* status, void* stream) {
    SX_REQUIRE(n_edges >= 0 && cap >= 1, "sx_cell_bvh_traverse_edges: bad sizes");
    if (n_edges == 0) return SX_OK;
    SX_REQUIRE(edges && p4 && grid8 && origin_box6 && nmin4 && nmax4 && prefix && face_rec8 && cand && num &&
                   status,
               "sx_cell_bvh_traverse_edges: null pointer");
    launch(cell_traverse_kernel<true>, traverse_grid(cell_traverse_kernel<true>, n_edges), CT_BLOCK, 0,
           as_stream(stream), n_edges,
           (const float4*)p4, padding, grid8, origin_box6, (const float4*)nmin4, (const float4*)nmax4, prefix,
           (const float4*)face_rec8, cap, cand, num, status, edges);
    return check_launch("cell_traverse_kernel");
}

extern "C" int sx_face_bvh_refit(int n, const int* sorted_ids, const float* fmin4, const float* fmax4,
                                 const int* child_a, const int* child_b, const int* parent, float* nmin4,
                                 float* nmax4, int* flags, int* status, void* stream) {
    SX_REQUIRE(n >= 1, "sx_face_bvh_refit: n must be >= 1");
    SX_REQUIRE(sorted_ids && fmin4 && fmax4 && parent && nmin4 && nmax4 && status &&
                   (n == 1 || (child_a && child_b && flags)),
               "sx_face_bvh_refit: null pointer");
    launch(face_refit_kernel, grid_for(n, 256), 256, 0, as_stream(stream), 
        n, sorted_ids, (const float4*)fmin4, (const float4*)fmax4, child_a, child_b, parent, (float4*)nmin4,
        (float4*)nmax4, flags, status);
    return check_launch("face_refit_kernel");
}

extern "C" int sx_face_bvh_refit_tiled(int n, const int* sorted_ids, const float* fmin4, const float* fmax4,
                                       const int* child_a, const int* child_b, const int* parent, const int* range_l,
                                       const int* range_r, float* nmin4, float* nmax4, int* flags, int* status,
                                       void* stream) {
    SX_REQUIRE(n >= 1, "sx_face_bvh_refit_tiled: n must be >= 1");
    SX_REQUIRE(sorted_ids && fmin4 && fmax4 && parent && nmin4 && nmax4 && status &&
                   (n == 1 || (child_a && child_b && flags && range_l && range_r)),
               "sx_face_bvh_refit_tiled: null pointer");
    launch(face_refit_tiled_kernel, grid_for(n, FR_TILE), FR_TILE, 0, as_stream(stream), n, sorted_ids,
           (const float4*)fmin4, (const float4*)fmax4, child_a, child_b, parent, range_l, range_r, (float4*)nmin4,
           (float4*)nmax4, flags, status);
    return check_launch("face_refit_tiled_kernel");
}

// aux: [level entries, 32 bytes each][n - 1 child records of 64 bytes]
extern "C" size_t sx_face_bvh_aux_bytes(int n) {
    return n < 1 ? 0 : (size_t)level_entries(n) * 32 + (size_t)n * 64;
}

extern "C" int sx_face_bvh_refit_ranges(int n, const int* sorted_ids, const float* fmin4, const float* fmax4,
                                        const int* range_l, const int* range_r, const int* parent, float* nmin4,
                                        float* nmax4, float* aux, size_t aux_bytes, void* stream) {
    SX_REQUIRE(n >= 1, "sx_face_bvh_refit_ranges: n must be >= 1");
    SX_REQUIRE(sorted_ids && fmin4 && fmax4 && nmin4 && nmax4 && aux && (n == 1 || (range_l && range_r && parent)),
               "sx_face_bvh_refit_ranges: null pointer");
    SX_REQUIRE(((uintptr_t)aux & 15) == 0 && aux_bytes >= sx_face_bvh_aux_bytes(n),
               "sx_face_bvh_refit_ranges: aux must be 16-byte aligned and sx_face_bvh_aux_bytes long");
    cudaStream_t s = as_stream(stream);
    const LevelTable t = level_table(n);
    float4 *lv = (float4*)aux, *rec = lv + 2 * level_entries(n);
    // blocks up to the padded end of level 1 (2), so that the padding gets written
    const long long cover =
        t.top < 1 ? n : t.top < 2 ? (t.count[1] + 7LL) / 8 * 64 : (t.count[2] + 7LL) / 8 * 512;
    launch(face_leaves_kernel, grid_for(cover, 256), 256, 0, s, n, sorted_ids, (const float4*)fmin4,
           (const float4*)fmax4, parent, range_l, (float4*)nmin4, (float4*)nmax4, lv, rec, t);
    int k = 3;
    for (; k <= t.top && t.count[k - 1] > 4096; ++k)
        launch(face_level_kernel, grid_for((t.count[k] + 7LL) / 8 * 64, 256), 256, 0, s, lv, t, k);
    if (k <= t.top) launch(face_top_levels_kernel, 1, 1024, 0, s, lv, t, k);
    if (n > 1)
        launch(face_ranges_kernel, grid_for(n - 1, 256), 256, 0, s, n, range_l, range_r, parent, (float4*)nmin4,
               (float4*)nmax4, (const float4*)lv, rec, t);
    return check_launch("sx_face_bvh_refit_ranges");
}

extern "C" int sx_face_bvh_query(int n, const float* p4, int n_queries, float padding, const int* sorted_ids,
                                 const float* nmin4, const float* nmax4, const float* aux, int cap, int* cand,
                                 int* num, int* status, const int* order, void* stream) {
    SX_REQUIRE(n >= 1 && n_queries >= 0 && cap >= 1, "sx_face_bvh_query: bad sizes");
    if (n_queries == 0) return SX_OK;
    SX_REQUIRE(p4 && sorted_ids && nmin4 && nmax4 && aux && cand && num && status, "sx_face_bvh_query: null pointer");
    launch(face_query_kernel, grid_for(n_queries, 128), 128, 0, as_stream(stream), n, n_queries, (const float4*)p4,
           padding, sorted_ids, (const float4*)nmin4, (const float4*)nmax4,
           (const float4*)aux + 2 * level_entries(n), cap, cand, num, status, order);
    return check_launch("face_query_kernel");
}

extern "C" int sx_face_bvh_traverse(int n, const float* p4, int n_queries, float padding, const int* child_a,
                                    const int* child_b, const int* sorted_ids, const float* nmin4,
                                    const float* nmax4, int cap, int* cand, int* num, int* status, void* stream) {
    SX_REQUIRE(n >= 1 && n_queries >= 0 && cap >= 1, "sx_face_bvh_traverse: bad sizes");
    if (n_queries == 0) return SX_OK;
    SX_REQUIRE(p4 && sorted_ids && nmin4 && nmax4 && cand && num && status && (n == 1 || (child_a && child_b)),
               "sx_face_bvh_traverse: null pointer");
    launch(face_traverse_kernel, grid_for(n_queries, 128), 128, 0, as_stream(stream), 
        n, n_queries, (const float4*)p4, padding, child_a, child_b, sorted_ids, (const float4*)nmin4,
        (const float4*)nmax4, cap, cand, num, status, (const int*)nullptr);
    return check_launch("face_traverse_kernel");
}

extern "C" int sx_face_bvh_traverse_ordered(int n, const float* p4, int n_queries, float padding,
                                            const int* child_a, const int* child_b, const int* sorted_ids,
                                            const float* nmin4, const float* nmax4, int cap, int* cand, int* num,
                                            int* status, const int* order, void* stream) {
    SX_REQUIRE(n >= 1 && n_queries >= 0 && cap >= 1, "sx_face_bvh_traverse_ordered: bad sizes");
    if (n_queries == 0) return SX_OK;
    SX_REQUIRE(p4 && sorted_ids && nmin4 && nmax4 && cand && num && status && order &&
                   (n == 1 || (child_a && child_b)),
               "sx_face_bvh_traverse_ordered: null pointer");
    launch(face_traverse_kernel, grid_for(n_queries, 128), 128, 0, as_stream(stream), n, n_queries,
           (const float4*)p4, padding, child_a, child_b, sorted_ids, (const float4*)nmin4, (const float4*)nmax4, cap,
           cand, num, status, order);
    return check_launch("face_traverse_kernel");
}
