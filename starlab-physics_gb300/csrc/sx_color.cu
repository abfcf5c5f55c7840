// Constraint-graph colouring (framework/utilities/graph_coloring.py).
//
// The reference builds a dense E x E adjacency (initAdjEdges :112-129) and
// colours edges sequentially, first-fit, in edge-id order (colorEdgesGreedy
// :131-149), then sorts edges by colour with a stable counting sort
// (colorCountingSort :172-201).  Here: a vertex -> edge incidence list replaces
// the dense matrix, and the sequential first-fit is reproduced exactly: an edge
// takes its colour as soon as every adjacent edge with a smaller id has one
// (those are exactly the edges a sequential pass would have coloured before it).
// One launch propagates colours from edge to edge along the vertices' lists
// (color_push_kernel); no host synchronisation.  The stable sort is the library's
// radix sort.
#include "sx_common.cuh"

extern "C" size_t sx_radix_sort_workspace_bytes(int n);
extern "C" int sx_radix_sort_pairs(unsigned* keys, int* vals, int n, int bits, void* ws, size_t ws_bytes,
                                   void* stream);

namespace sx {

constexpr int kMaxColorWords = 4;  // up to 128 colours

static inline size_t a256(size_t b) { return (b + 255) & ~(size_t)255; }

__global__ void inc_count_kernel(int E, const int* __restrict__ edges, int* cnt) {
    pdl_entry();
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    atomicAdd(cnt + edges[2 * e], 1);
    atomicAdd(cnt + edges[2 * e + 1], 1);
}

__global__ void inc_fill_kernel(int E, const int* __restrict__ edges, const int* __restrict__ ptr, int* cursor,
                                int* inc) {
    pdl_entry();
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    int a = edges[2 * e], b = edges[2 * e + 1];
    inc[ptr[a] + atomicAdd(cursor + a, 1)] = e;
    inc[ptr[b] + atomicAdd(cursor + b, 1)] = e;
}

// ---------------------------------------------------------------------------
// Propagation.  The edges at a vertex, in id order, form a chain: when one has
// its colour, so have all lower ones, so an edge depends only on its
// predecessor at either endpoint, and one message per endpoint -- the set of
// colours used at that vertex so far -- tells its successor all it needs.  A
// thread that colours an edge sends its two messages; the message that completes
// an edge makes it ready, and the sender queues it with both sets.
//
// A block works through a ring of ready edges in shared memory, all threads
// taking one per step; it starts from edges without predecessors (seeds).
// Blocks never wait for one another; one whose ring is full leaves the rest to
// color_edges_kernel (*spill != 0).  Two forms, told apart by the number of
// seeds:
//
// * few seeds (a sheet numbered row by row has one): color_chain_kernel, a
//   single block, since the chain of dependent edges is the limit and not the
//   width (the 256 x 256 sheet's 195 388 edges: 2 037 steps, up to 170 edges
//   wide).  Only the messages under way have to be kept, up to two per edge of
//   the front, so they live in a hash table in shared memory, and those that find
//   their bucket full in global memory.
// * many seeds (concatenated sheets, shuffled numbering): color_push_kernel,
//   every SM.  Messages are 64-bit atomic adds on the edge's word, and the add
//   that completes the word returns both sets; a link costs an atomic's round
//   trip and the ring's bookkeeping, 1.5 us.  The seeds are dealt evenly to the
//   blocks: a block that runs dry ends, so with those of a range of edges each the
//   work came down to a few blocks (us; dealt / by ranges / color_edges_kernel
//   alone: 195 585 edges of a sheet in random order 212 / 432 / 261, an icosphere's
//   122 880 226 / 539 / 278, 1000 8 x 8 sheets 195 / 205 / 369).
//
// The former form, in which each edge's thread waited for the one neighbour that
// blocked it and then read all neighbours' colours again, took 3 us a link.
//
// A step of the single block takes 0.85 us: the successors' own successors come
// from L2 (prefetching or loading their lines a step ahead made it slower), then
// a barrier, the table and the ring.  With the messages in global memory it took
// 1 us (plain stores: a line just stored misses L1), with atomics 1.5 us.  Sheets
// of 256 x 256 / 512 x 512 / 1024 x 1024, ms: 1.75 / 4.0 / 10.7, with bending pairs
// 2.4 / 6.0 / 21.6; a table that lost the messages of a full bucket, and left the
// rest to color_edges_kernel, took 1.78 / 4.6 / 17 to 57 and 2.6 / 26 / 116.
//
// A message: bits 0-29 colours 0-29, bit 30: a higher colour is among them and
// the whole set is in msg.  Word of an edge: bits 0-30 the message at endpoint
// 0, 31-61 at endpoint 1, 62-63 the messages that need not come plus those that
// came (2 = ready).  Successor slot: 4 * edge + 2 (it has no predecessor at its
// other endpoint: one message makes it ready) + the endpoint, or kNone.
// ---------------------------------------------------------------------------
constexpr int CP_THREADS = 256, CP_RING = 4096;
constexpr int CP_BUCKETS = 2048;  // of four messages each
constexpr unsigned kNone = 0xffffffffu;
constexpr unsigned kMsgLow = 0x3fffffffu, kMsgMore = 0x40000000u;
constexpr int kManySeeds = 64;

// Chains: waits[e] bit s: edge e has a predecessor at endpoint s.  An edge (v, v)
// counts as having endpoint 0 only.
__global__ void color_waits_kernel(int E, const int* __restrict__ edges, const int* __restrict__ ptr,
                                   const int* __restrict__ inc, uint2* __restrict__ succ,
                                   unsigned long long* __restrict__ word, unsigned char* __restrict__ waits,
                                   int* __restrict__ color, int* __restrict__ ids, int* __restrict__ n_seeds,
                                   int* __restrict__ seeds) {
    pdl_entry();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const int a = edges[2 * e], b = edges[2 * e + 1];
    unsigned next[2] = {kNone, kNone};
    int w = 0;
    for (int s = 0; s < (a == b ? 1 : 2); ++s) {
        const int v = s ? b : a;
        int best = 0x7fffffff;
        for (int k = ptr[v]; k < ptr[v + 1]; ++k) {
            const int o = inc[k];
            if (o > e) best = min(best, o);
            if (o < e) w |= 1 << s;
        }
        if (best != 0x7fffffff) next[s] = 4u * (unsigned)best + (edges[2 * best] == v ? 0u : 1u);
    }
    succ[e] = make_uint2(next[0], next[1]);
    waits[e] = (unsigned char)w;
    word[e] = (unsigned long long)(2 - __popc(w)) << 62;
    color[e] = -1;
    ids[e] = e;
    if (w == 0) seeds[atomicAdd(n_seeds, 1)] = e;
}
__global__ void color_lone_kernel(int E, uint2* __restrict__ succ, const unsigned char* __restrict__ waits) {
    pdl_entry();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    uint2 s = succ[e];
    if (s.x != kNone && waits[s.x >> 2] != 3) s.x |= 2u;
    if (s.y != kNone && waits[s.y >> 2] != 3) s.y |= 2u;
    succ[e] = s;
}

__device__ __forceinline__ uint4 message_set(unsigned m, const uint4* msg) {
    if (m & kMsgMore) return __ldcg(msg);
    return make_uint4(m & kMsgLow, 0u, 0u, 0u);
}
__device__ __forceinline__ void add_color(uint4* s, int c) {
    const unsigned bit = 1u << (c & 31);
    if (c < 32) s->x |= bit;
    else if (c < 64) s->y |= bit;
    else if (c < 96) s->z |= bit;
    else s->w |= bit;
}
// smallest colour outside both sets, 0 when there is none below max_colors
__device__ __forceinline__ int first_free(uint4 a, uint4 b, int max_colors) {
    const unsigned w[4] = {a.x | b.x, a.y | b.y, a.z | b.z, a.w | b.w};
    int c = 0x7fffffff;
#pragma unroll
    for (int i = 3; i >= 0; --i)
        if (w[i] != 0xffffffffu) c = 32 * i + __ffs(~w[i]) - 1;
    return c < max_colors ? c : 0;
}
// Colours edge e given its two messages and turns them into the messages for
// its successors (slots s.x and s.y, -1: none), whose whole sets go to msg when
// they hold colours from 30 on.
__device__ __forceinline__ size_t msg_index(unsigned s) { return 2 * (size_t)(s >> 2) + (s & 1u); }
__device__ __forceinline__ int color_edge(int e, unsigned* ma, unsigned* mb, uint2 s, uint4* msg, int max_colors) {
    const unsigned used = *ma | *mb;
    const int low = __ffs(~used) - 1;
    if (!(used & kMsgMore) && low < 30 && low < max_colors) {
        *ma |= 1u << low;
        *mb |= 1u << low;
        return low;
    }
    uint4 a = message_set(*ma, msg + 2 * (size_t)e), b = message_set(*mb, msg + 2 * (size_t)e + 1);
    const int c = first_free(a, b, max_colors);
    add_color(&a, c);
    add_color(&b, c);
    *ma = a.x & kMsgLow;
    *mb = b.x & kMsgLow;
    if ((a.x & ~kMsgLow) | a.y | a.z | a.w) {
        if (s.x != kNone) msg[msg_index(s.x)] = a;
        *ma |= kMsgMore;
    }
    if ((b.x & ~kMsgLow) | b.y | b.z | b.w) {
        if (s.y != kNone) msg[msg_index(s.y)] = b;
        *mb |= kMsgMore;
    }
    return c;
}
// appends the edges behind successor slots s.x (if r0) and s.y (if r1), with
// their successors and messages, to the ring: one atomic per warp
__device__ __forceinline__ void ring_push(int4* ring, unsigned* ring_b, int* s_tail, bool r0, bool r1, uint2 s,
                                          uint2 n0, uint2 n1, uint2 m0, uint2 m1) {
    const int lane = threadIdx.x & 31;
    const unsigned q0 = __ballot_sync(0xffffffffu, r0), q1 = __ballot_sync(0xffffffffu, r1);
    if ((q0 | q1) == 0u) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(s_tail, __popc(q0) + __popc(q1));
    at = __shfl_sync(0xffffffffu, at, 0);
    const unsigned below = (1u << lane) - 1u;
    if (r0) {
        const int i = (at + __popc(q0 & below)) & (CP_RING - 1);
        ring[i] = make_int4((int)(s.x >> 2), (int)n0.x, (int)n0.y, (int)m0.x);
        ring_b[i] = m0.y;
    }
    if (r1) {
        const int i = (at + __popc(q0) + __popc(q1 & below)) & (CP_RING - 1);
        ring[i] = make_int4((int)(s.y >> 2), (int)n1.x, (int)n1.y, (int)m1.x);
        ring_b[i] = m1.y;
    }
}
// n edges leave the ring and, past a barrier, at most 2 n enter it (n < 0: held < 0)
__device__ __forceinline__ int ring_take(int held, int threads) {
    return min(min(held, threads), CP_RING - max(held, 0));
}

// The messages under way: {edge + 1, message} in the edge's bucket, 0 when free.  A
// step looks up the partners of all its messages (and takes out those found), then,
// past a barrier, enters the messages without one: two sent in the same step meet
// there, since both walk the bucket from its start and nothing is taken out
// meanwhile.  A message that finds its bucket full is parked in the edge's word in
// global memory, where its partner, which finds the bucket full in the same step,
// or parked[bucket] above 0 in a later one, meets it.
__device__ __forceinline__ int bucket_of(unsigned f) { return (int)((f * 2654435761u) >> 21); }
static_assert(CP_BUCKETS == 1 << 11, "bucket_of keeps 11 bits");
constexpr unsigned long long kParked = 1ull << 62;  // (word of an edge that waits for two messages: 0 before)
constexpr int kSomeParked = (int)0x80000000u;       // in the ring's tail: messages have been parked

__device__ __forceinline__ bool table_take(unsigned long long* table, unsigned s, unsigned* other) {
    const unsigned f = s >> 2;
    unsigned long long* bucket = table + 4 * bucket_of(f);
    const ulonglong2* two = reinterpret_cast<const ulonglong2*>(bucket);
    const ulonglong2 p = two[0], q = two[1];
    const unsigned long long v[4] = {p.x, p.y, q.x, q.y};
    int at = -1;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if ((unsigned)(v[i] >> 32) == f + 1u) {
            *other = (unsigned)v[i] & 0x7fffffffu;
            at = i;
        }
    const bool found = at >= 0;
    if (found) bucket[at] = 0ull;
    return found;
}
__device__ __forceinline__ bool parked_take(int* parked, const unsigned long long* word, unsigned s, unsigned* other) {
    const unsigned f = s >> 2;
    int* count = parked + bucket_of(f);
    if (*count <= 0) return false;
    const unsigned long long v = __ldcg(word + f);
    if (!(v & kParked)) return false;
    *other = (unsigned)v & 0x7fffffffu;
    atomicSub(count, 1);
    return true;
}
// >= 0: entry of the partner, which also entered in this step; -1: entered; -2: bucket full
__device__ __forceinline__ int table_enter(unsigned long long* table, unsigned s, unsigned m, unsigned* other) {
    const unsigned f = s >> 2;
    const int b = 4 * bucket_of(f);
    const unsigned long long mine = ((unsigned long long)(f + 1u) << 32) | m;
    for (int i = 0; i < 4; ++i) {
        const unsigned long long old = atomicCAS(table + b + i, 0ull, mine);
        if (old == 0ull) return -1;
        if ((unsigned)(old >> 32) == f + 1u) {
            *other = (unsigned)old & 0x7fffffffu;
            return b + i;
        }
    }
    return -2;
}
// Parks a message; whether its partner stands there from this step
__device__ __forceinline__ bool park(int* parked, unsigned long long* word, int* s_tail, unsigned s, unsigned m,
                                     unsigned* other) {
    const unsigned f = s >> 2;
    const unsigned long long old = atomicCAS(word + f, 0ull, kParked | m);
    atomicAdd(parked + bucket_of(f), old == 0ull ? 1 : -1);
    atomicOr(s_tail, kSomeParked);
    if (old != 0ull) *other = (unsigned)old & 0x7fffffffu;
    return old != 0ull;
}

struct Chain {
    const uint2* succ;
    unsigned long long* word;
    uint4* msg;
    int max_colors;
    int *color, *spill;
    int4* ring;  // {edge, successor slots, message 0}
    unsigned* ring_b;  // message 1
    unsigned long long* table;
    int *parked, *s_tail;
};
// Steps until the ring is empty or full, and without PARKED until a message has been
// parked (the loop of its own saves a step the look at parked, 8 % of it).
template <int THREADS, bool PARKED>
__device__ __forceinline__ void chain_steps(const Chain& c, int& head, int& done0, int& done1) {
    const int tid = threadIdx.x;
    for (;;) {
        __syncthreads();
        const int tail = *c.s_tail;
        const int held = (PARKED ? tail & ~kSomeParked : tail) - head, n = ring_take(held, THREADS);
        if (n <= 0) {  // (without PARKED held is below 0 from then on)
            if (held > 0 && tid == 0) atomicOr(c.spill, 1);
            break;
        }
        // partners that met while entering in the last step
        if (done0 >= 0) c.table[done0] = 0ull;
        if (done1 >= 0) c.table[done1] = 0ull;
        done0 = done1 = -1;
        uint2 s = make_uint2(kNone, kNone), n0 = s, n1 = s;
        unsigned ma = 0u, mb = 0u, oa = 0u, ob = 0u;
        bool r0 = false, r1 = false;
        if (tid < n) {
            const int at = (head + tid) & (CP_RING - 1);
            const int4 r = c.ring[at];
            ma = (unsigned)r.w;
            mb = c.ring_b[at];
            s = make_uint2((unsigned)r.y, (unsigned)r.z);
            if (s.x != kNone) n0 = __ldg(c.succ + (s.x >> 2));
            if (s.y != kNone) n1 = __ldg(c.succ + (s.y >> 2));
            c.color[r.x] = color_edge(r.x, &ma, &mb, s, c.msg, c.max_colors);
            if (s.x != kNone) r0 = (s.x & 2u) || table_take(c.table, s.x, &oa);
            if (s.y != kNone) r1 = (s.y & 2u) || table_take(c.table, s.y, &ob);
            if (PARKED) {
                if (s.x != kNone && !r0) r0 = parked_take(c.parked, c.word, s.x, &oa);
                if (s.y != kNone && !r1) r1 = parked_take(c.parked, c.word, s.y, &ob);
            }
        }
        head += n;
        __syncthreads();
        if (s.x != kNone && !r0) {
            done0 = table_enter(c.table, s.x, ma, &oa);
            r0 = done0 >= 0;
            if (done0 == -2) r0 = park(c.parked, c.word, c.s_tail, s.x, ma, &oa);
        }
        if (s.y != kNone && !r1) {
            done1 = table_enter(c.table, s.y, mb, &ob);
            r1 = done1 >= 0;
            if (done1 == -2) r1 = park(c.parked, c.word, c.s_tail, s.y, mb, &ob);
        }
        ring_push(c.ring, c.ring_b, c.s_tail, r0, r1, s, n0, n1, (s.x & 1u) ? make_uint2(oa, ma) : make_uint2(ma, oa),
                  (s.y & 1u) ? make_uint2(ob, mb) : make_uint2(mb, ob));
    }
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) color_chain_kernel(const uint2* __restrict__ succ, unsigned long long* word,
                                                              uint4* msg, int max_colors, int* color,
                                                              const int* __restrict__ n_seeds,
                                                              const int* __restrict__ seeds, int* spill) {
    pdl_entry();
    const int ns = *n_seeds;
    if (ns > kManySeeds) return;
    extern __shared__ int4 ring[];
    __shared__ int s_tail;
    Chain c{succ, word, msg, max_colors, color, spill, ring};
    c.ring_b = reinterpret_cast<unsigned*>(ring + CP_RING);
    c.table = reinterpret_cast<unsigned long long*>(c.ring_b + CP_RING);
    c.parked = reinterpret_cast<int*>(c.table + 4 * CP_BUCKETS);
    c.s_tail = &s_tail;
    const int tid = threadIdx.x;
    for (int i = tid; i < 4 * CP_BUCKETS; i += THREADS) c.table[i] = 0ull;
    for (int i = tid; i < CP_BUCKETS; i += THREADS) c.parked[i] = 0;
    if (tid == 0) s_tail = ns;
    if (tid < ns) {
        const uint2 s = __ldg(succ + seeds[tid]);
        c.ring[tid] = make_int4(seeds[tid], (int)s.x, (int)s.y, 0);
        c.ring_b[tid] = 0u;
    }
    int head = 0, done0 = -1, done1 = -1;
    chain_steps<THREADS, false>(c, head, done0, done1);
    __syncthreads();
    if (s_tail < 0) chain_steps<THREADS, true>(c, head, done0, done1);
}

// adds a message to successor slot s; the successor's word afterwards
__device__ __forceinline__ unsigned long long color_send(unsigned s, unsigned m, unsigned long long* word) {
    if (m & kMsgMore) __threadfence();  // after the store of the whole set
    const unsigned long long add = ((unsigned long long)m << (31 * (s & 1u))) + (1ull << 62);
    return atomicAdd(word + (s >> 2), add) + add;
}

__global__ void __launch_bounds__(CP_THREADS) color_push_kernel(int E, const uint2* __restrict__ succ,
                                                                unsigned long long* word, uint4* msg, int max_colors,
                                                                int* color, const int* __restrict__ n_seeds,
                                                                const int* __restrict__ seeds, int* spill) {
    pdl_entry();
    const int ns = *n_seeds;
    if (ns <= kManySeeds) return;
    extern __shared__ int4 ring[];  // {edge, successor slots, message 0}
    unsigned* ring_b = reinterpret_cast<unsigned*>(ring + CP_RING);  // message 1
    __shared__ int s_tail;
    const int tid = threadIdx.x;
    if (tid == 0) s_tail = 0;
    const int share = (ns + (int)gridDim.x - 1) / (int)gridDim.x;
    int scan = (int)min((long long)blockIdx.x * share, (long long)ns);
    const int hi = min(scan + share, ns);
    int head = 0;  // uniform; head and tail count up to E at most
    for (;;) {
        __syncthreads();
        int tail = s_tail;
        // the block's seeds, while there is room
        while (scan < hi && tail - head <= CP_RING / 2 - CP_THREADS) {
            __syncthreads();
            const bool seed = scan + tid < hi;
            const int e = seed ? seeds[scan + tid] : 0;
            const uint2 none = make_uint2(kNone, kNone), zero = make_uint2(0u, 0u);
            ring_push(ring, ring_b, &s_tail, seed, false, make_uint2(4u * (unsigned)e, kNone), seed ? succ[e] : none,
                      none, zero, zero);
            scan += CP_THREADS;
            __syncthreads();
            tail = s_tail;
        }
        const int held = tail - head, n = ring_take(held, CP_THREADS);
        if (n == 0) {
            if (held > 0 && tid == 0) atomicOr(spill, 1);
            break;
        }
        uint2 s = make_uint2(kNone, kNone), n0 = s, n1 = s;
        int4 r = make_int4(-1, -1, -1, 0);
        unsigned mb = 0u;
        if (tid < n) {
            r = ring[(head + tid) & (CP_RING - 1)];
            mb = ring_b[(head + tid) & (CP_RING - 1)];
            s = make_uint2((unsigned)r.y, (unsigned)r.z);
        }
        head += n;
        __syncthreads();
        unsigned long long w0 = 0, w1 = 0;
        if (r.x >= 0) {
            unsigned ma = (unsigned)r.w;
            if ((ma | mb) & kMsgMore) __threadfence();  // before the loads of the whole sets
            color[r.x] = color_edge(r.x, &ma, &mb, s, msg, max_colors);
            if (s.x != kNone) {
                w0 = color_send(s.x, ma, word);
                n0 = __ldg(succ + (s.x >> 2));
            }
            if (s.y != kNone) {
                w1 = color_send(s.y, mb, word);
                n1 = __ldg(succ + (s.y >> 2));
            }
        }
        const auto both = [](unsigned long long w) {
            return make_uint2((unsigned)w & 0x7fffffffu, (unsigned)(w >> 31) & 0x7fffffffu);
        };
        ring_push(ring, ring_b, &s_tail, (w0 >> 62) == 2, (w1 >> 62) == 2, s, n0, n1, both(w0), both(w1));
    }
}

// Tries to colour edge e: false if an adjacent edge with a smaller id has no
// colour yet; otherwise e gets the smallest colour none of them has (or keeps
// the one it has).  Colours once set never change, so reading a neighbour's
// colour set earlier in the same round gives the same choice.
__device__ __forceinline__ bool color_try(int e, const int* __restrict__ edges, const int* __restrict__ ptr,
                                          const int* __restrict__ inc, int max_colors, int* color, int* blocker) {
    volatile int* vc = color;
    if (vc[e] >= 0) return true;
    unsigned forbid[kMaxColorWords] = {0u, 0u, 0u, 0u};
    for (int s = 0; s < 2; ++s) {
        const int v = edges[2 * e + s];
        for (int k = ptr[v]; k < ptr[v + 1]; ++k) {
            const int o = inc[k];
            if (o >= e) continue;
            const int c = vc[o];
            if (c < 0) {
                *blocker = o;
                return false;
            }
            forbid[c >> 5] |= 1u << (c & 31);
        }
    }
    int pick = 0;
    for (int c = 0; c < max_colors; ++c) {
        if (!(forbid[c >> 5] & (1u << (c & 31)))) {
            pick = c;
            break;
        }
    }
    vc[e] = pick;
    return true;
}

// What color_push_kernel left, in one cooperative launch (all threads resident):
// a thread takes its edges in ascending id order (grid stride) and colours each
// as soon as every adjacent edge with a smaller id has a colour.  The smallest
// uncoloured edge never waits (its thread has finished all its smaller edges),
// so the colouring always progresses.  A thread gathers the ids of its edge's
// lower neighbours once (up to kMaxLower; more falls back to color_try's
// sequential scan), then reads all their colours with independent loads, and
// when one is missing waits on that neighbour alone, re-reading with a short
// sleep.  Each wait is bounded: after kColorPolls re-reads the edge stays
// uncoloured and SX_STATUS_WAIT_TIMEOUT is set, which makes the edges waiting
// on it give up in turn.
constexpr int kColorPolls = 1 << 21;
constexpr int kMaxLower = 24;

__global__ void __launch_bounds__(256, 4) color_edges_kernel(int E, const int* __restrict__ edges,
                                                          const int* __restrict__ ptr, const int* __restrict__ inc,
                                                          int max_colors, int* color, int* status,
                                                          const int* __restrict__ spill) {
    pdl_entry();
    if (*spill == 0) return;
    const long long stride = (long long)gridDim.x * blockDim.x;
    volatile int* vc = color;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
        if (vc[e] >= 0) continue;
        int polls = 0;
        bool timed_out = false;
        // the lower neighbours of e, once
        int nb[kMaxLower];
        int n = 0;
        bool many = false;
        for (int s = 0; s < 2; ++s) {
            const int v = edges[2 * e + s];
            for (int k = ptr[v]; k < ptr[v + 1]; ++k) {
                const int o = inc[k];
                if (o >= e) continue;
                if (n < kMaxLower) {
                    nb[n++] = o;
                } else {
                    many = true;
                }
            }
        }
        if (many) {
            int blocker = -1;
            bool done = false;
            while (!done && !timed_out) {
                done = color_try((int)e, edges, ptr, inc, max_colors, color, &blocker);
                const volatile int* vb = color + blocker;
                while (!done && *vb < 0) {
                    if (++polls > kColorPolls) {
                        timed_out = true;
                        break;
                    }
                    __nanosleep(32);
                }
            }
        } else {
            for (;;) {
                int c[kMaxLower];
#pragma unroll
                for (int j = 0; j < kMaxLower; ++j) c[j] = j < n ? vc[nb[j]] : 0;
                int blocker = -1;
                unsigned forbid[kMaxColorWords] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int j = 0; j < kMaxLower; ++j) {
                    if (j < n) {
                        if (c[j] < 0) {
                            if (blocker < 0) blocker = nb[j];
                        } else {
                            forbid[c[j] >> 5] |= 1u << (c[j] & 31);
                        }
                    }
                }
                if (blocker < 0) {
                    int pick = 0;
                    for (int q = 0; q < max_colors; ++q) {
                        if (!(forbid[q >> 5] & (1u << (q & 31)))) {
                            pick = q;
                            break;
                        }
                    }
                    vc[e] = pick;
                    break;
                }
                const volatile int* vb = color + blocker;
                while (*vb < 0) {
                    if (++polls > kColorPolls) {
                        timed_out = true;
                        break;
                    }
                    __nanosleep(32);
                }
                if (timed_out) break;
            }
        }
        if (timed_out) atomicOr(status, SX_STATUS_WAIT_TIMEOUT);
    }
}

// counts per block first: a sheet has a dozen colours, and 195 585 atomics on
// their words took 36 us
__global__ void __launch_bounds__(256) color_hist_kernel(int E, const int* __restrict__ color, unsigned* keys,
                                                         unsigned* hist) {
    pdl_entry();
    __shared__ unsigned cnt[128];
    if (threadIdx.x < 128) cnt[threadIdx.x] = 0u;
    __syncthreads();
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (long long)gridDim.x * blockDim.x) {
        const int c = color[e];  // -1 only if a bounded wait gave up (status bit set)
        keys[e] = c < 0 ? 255u : (unsigned)c;
        if (c >= 0) atomicAdd(cnt + c, 1u);
    }
    __syncthreads();
    if (threadIdx.x < 128 && cnt[threadIdx.x] != 0u) atomicAdd(hist + threadIdx.x, cnt[threadIdx.x]);
}

// exclusive scan of the colour histogram (max_colors <= 128) -> start offsets
__global__ void __launch_bounds__(128) color_prefix_kernel(int max_colors, const unsigned* hist, int* prefix) {
    pdl_entry();
    __shared__ unsigned wsum[4];
    const int t = threadIdx.x, lane = t & 31;
    const unsigned v = t < max_colors ? hist[t] : 0u;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) wsum[t >> 5] = incl;
    __syncthreads();
    for (int w = 0; w < t >> 5; ++w) incl += wsum[w];
    if (t < max_colors) prefix[t] = (int)(incl - v);
}

}  // namespace sx

using namespace sx;

// workspace: [status, spill, seed count][ptr V+1][cursor V][inc 2E][succ E][word E][waits E][msg 2E][keys E][hist 128][radix ws E]
extern "C" size_t sx_color_workspace_bytes(int n_verts, int n_edges) {
    size_t V = (size_t)(n_verts > 0 ? n_verts : 1), E = (size_t)(n_edges > 0 ? n_edges : 1);
    return 1024 + a256((V + 1) * 4) + a256(V * 4) + a256(2 * E * 4) + a256(E * 8) + a256(E * 8) + a256(E) +
           a256(2 * E * 16) + a256(E * 4) + a256(128 * 4) + sx_radix_sort_workspace_bytes(n_edges);
}

extern "C" int sx_color_edges_greedy(const int* edges, int n_edges, int n_verts, int max_colors, int* color,
                                     int* sorted_edges, int* prefix, void* ws, size_t ws_bytes, void* stream) {
    SX_REQUIRE(n_edges >= 0 && n_verts >= 0, "sx_color_edges_greedy: bad sizes");
    SX_REQUIRE(max_colors >= 1 && max_colors <= 32 * kMaxColorWords, "sx_color_edges_greedy: max_colors in [1, 128]");
    SX_REQUIRE(prefix, "sx_color_edges_greedy: null prefix");
    cudaStream_t s = as_stream(stream);
    if (n_edges == 0) {
        SX_CUDA(cudaMemsetAsync(prefix, 0, sizeof(int) * max_colors, s));
        return SX_OK;
    }
    SX_REQUIRE(edges && color && sorted_edges, "sx_color_edges_greedy: null pointer");
    SX_REQUIRE(ws && ws_bytes >= sx_color_workspace_bytes(n_verts, n_edges),
               "sx_color_edges_greedy: workspace too small");
    const size_t V = (size_t)(n_verts > 0 ? n_verts : 1), E = (size_t)n_edges;
    int* status = (int*)ws;
    int *spill = status + 1, *n_seeds = status + 2;
    char* p = (char*)(((uintptr_t)(n_seeds + 1) + 255) & ~(uintptr_t)255);
    int* ptr = (int*)p; p += a256((V + 1) * 4);
    int* cursor = (int*)p; p += a256(V * 4);
    int* inc = (int*)p; p += a256(2 * E * 4);
    uint2* succ = (uint2*)p; p += a256(E * 8);
    unsigned long long* word = (unsigned long long*)p; p += a256(E * 8);
    unsigned char* waits = (unsigned char*)p; p += a256(E);
    uint4* msg = (uint4*)p; p += a256(2 * E * 16);
    unsigned* keys = (unsigned*)p; p += a256(E * 4);
    unsigned* hist = (unsigned*)p; p += a256(128 * 4);
    void* rws = p;
    int* seeds = (int*)keys;  // until the colours' keys are written

    // status, spill, ptr and cursor lie together at the start
    SX_CUDA(cudaMemsetAsync(ws, 0, (size_t)((char*)(cursor + V) - (char*)ws), s));
    launch(inc_count_kernel, grid_for(n_edges, 256), 256, 0, s, n_edges, edges, ptr);
    int rc = scan_u32(reinterpret_cast<unsigned*>(ptr), n_verts + 1, 0, s);
    if (rc) return rc;
    launch(inc_fill_kernel, grid_for(n_edges, 256), 256, 0, s, n_edges, edges, ptr, cursor, inc);
    launch(color_waits_kernel, grid_for(n_edges, 256), 256, 0, s, n_edges, edges, (const int*)ptr, (const int*)inc,
           succ, word, waits, color, sorted_edges, n_seeds, seeds);
    launch(color_lone_kernel, grid_for(n_edges, 256), 256, 0, s, n_edges, succ, (const unsigned char*)waits);
    constexpr size_t smem = (size_t)CP_RING * (sizeof(int4) + sizeof(unsigned));
    constexpr size_t smem_table = smem + CP_BUCKETS * (4 * sizeof(unsigned long long) + sizeof(int));
    // as many threads as a sheet of that many edges has edges ready at once (64 x 64: 60,
    // 256 x 256: 170 to 255, 512 x 512 with bending pairs: 770); a step of more threads
    // costs more.  256 / 512 / 1024 threads, ms, the two numberings of a sheet that the
    // package makes: 195 585 edges 1.75 / 1.85 / 2.03 and 1.39 / 1.46 / 1.58, 390 150
    // 2.33 / 2.42 / 2.58 and 2.54 / 2.05 / 2.17, 1 566 726 9.2 / 6.0 / 6.2 and 9.8 / 7.4 /
    // 8.0, 3 141 633 17.4 / 11.2 / 10.7 and 17.5 / 11.9 / 10.6
    const int chain_threads = n_edges <= 350000 ? 256 : n_edges <= 2500000 ? 512 : 1024;
    const auto chain = chain_threads == 256   ? color_chain_kernel<256>
                       : chain_threads == 512 ? color_chain_kernel<512>
                                              : color_chain_kernel<1024>;
    SX_CUDA(cudaFuncSetAttribute(chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_table));
    SX_CUDA(cudaFuncSetAttribute(color_push_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch(chain, 1, chain_threads, smem_table, s, (const uint2*)succ, word, msg, max_colors, color,
           (const int*)n_seeds, (const int*)seeds, spill);
    const int blocks = grid_for(n_edges, 4 * CP_THREADS);  // one block per SM at most
    launch(color_push_kernel, blocks < 152 ? blocks : 152, CP_THREADS, smem, s, n_edges, (const uint2*)succ, word, msg, max_colors, color, (const int*)n_seeds, (const int*)seeds, spill);
    rc = check_launch("colour propagation");
    if (rc) return rc;
    // every block resident (its threads wait on one another)
    {
        const int cap = resident_blocks(color_edges_kernel, 256);
        const int g = grid_for(n_edges, 256) < cap ? grid_for(n_edges, 256) : cap;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(g);
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        SX_CUDA(cudaLaunchKernelEx(&cfg, color_edges_kernel, n_edges, edges, (const int*)ptr, (const int*)inc,
                                   max_colors, color, status, (const int*)spill));
        note_launch();
    }
    SX_CUDA(cudaMemsetAsync(hist, 0, 128 * 4, s));
    const int hb = grid_for(n_edges, 1024);
    launch(color_hist_kernel, hb < 304 ? hb : 304, 256, 0, s, n_edges, (const int*)color, keys, hist);
    launch(color_prefix_kernel, 1, 128, 0, s, max_colors, (const unsigned*)hist, prefix);
    rc = check_launch("colour histogram");
    if (rc) return rc;
    return sx_radix_sort_pairs(keys, sorted_edges, n_edges, 8, rws, sx_radix_sort_workspace_bytes(n_edges), s);
}
