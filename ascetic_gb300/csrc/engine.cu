// The out-of-GPU-memory iteration engine: frontier kernels for BFS, SSSP, CC
// and PageRank over a device-resident static prefix of the edge array plus
// on-demand edges read straight from pinned host memory.
//
// What each iteration does, against the reference driver (CalculateOpt.cu:60-191):
//  - split of the active set into static and on-demand vertices, compaction
//    into lists, and the active counts (setStaticAndOverloadLabelBool,
//    thrust::reduce/exclusive_scan, setStaticActiveNodeArray,
//    setOverloadNodePointerSwap, gpu_kernels.cu:111-122, gpu_kernels.cuh:411-438)
//    happen here as a by-product of relaxation: the thread that lowers a value
//    and wins the vertex's bit in the next-frontier bitmap appends it, with one
//    warp-aggregated atomic per warp, to the static list, the on-demand list,
//    or (long lists) the segment list;
//  - the host gather of on-demand edges and the partitioned H2D copies
//    (GraphMeta.cuh:469-578, CalculateOpt.cu:146-178) are replaced by the
//    on-demand expansion kernel reading each active list directly from the
//    mapped pinned copy over the host link, so only active edges cross it;
//  - relaxation rules are those of bfs_kernelStatic / sssp_kernel /
//    cc_kernelStaticSwap (gpu_kernels.cuh:376-505, 441-481): atomicMin of
//    val[u]+1, val[u]+w, val[u]; PageRank sums follow prSumKernel_* and
//    prKernel_Opt (gpu_kernels.cuh:533-594).
//
// Load balance: each expansion launch is a persistent grid pulling work items
// from an atomic cursor. A work item of a sparse frontier is a tile of up to 256
// list entries (the CTA scans their degrees and walks the tile's concatenated edge
// range, so consecutive threads read consecutive column indices) or one segment of
// a vertex whose degree exceeds the huge-degree threshold (a CTA-wide stride over up
// to segment_edges edges of that list). A dense one is walked in id order, by merge
// items of 2048 rows plus edges or by tiles of 256 vertices (by_items).
#include <cooperative_groups.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <memory>
#include <new>
#include <mutex>
#include <thread>
#include <vector>
#include <string>
#include <sys/stat.h>

#include "common.h"

namespace asc {

namespace {

constexpr unsigned kFull = 0xffffffffu;
// Minimum resident CTAs per SM asked of the expansion kernels (register cap):
// 8 x 256 threads fill an SM, 32 registers each. Measured on RMAT scale 24 with
// bit-packed edges: 65.6 GTEPS at 8, 64.5 at 6, 57.3 at 4 (64 registers, half
// the warps: the loads over the host link want every warp the SM can hold).
// The same for the list-driven PageRank pull. The batched SSSP kernel takes 5 (48
// registers; at 6 or 8 it spills more than a few bytes). Kernels that hold a merge
// item in shared memory name their own: 6 (ASC_TRAV_BLOCKS, ASC_PR_ITEM_BLOCKS,
// ASC_MS_BFS_BLOCKS; 40 registers) or 4 (ASC_PR_SCATTER_BLOCKS).
#ifndef ASC_PR_MIN_BLOCKS
#define ASC_PR_MIN_BLOCKS 8
#endif
#ifndef ASC_MS_MIN_BLOCKS
#define ASC_MS_MIN_BLOCKS 5
#endif
#ifndef ASC_EXPAND_MIN_BLOCKS
#define ASC_EXPAND_MIN_BLOCKS 8
#endif
constexpr int kWarps = kBlock / 32;

// Self-checking build (nvcc -DASC_SELF_CHECK): indices the kernels take from
// device data (frontier lists, segment items, decoded edges, level-plane
// pointers, list and segment capacities) are checked before use; the first bad
// one is recorded as (site << 32 | index), its access is skipped, and the run
// or batch iteration that launched the kernel fails with ASC_ERR_CUDA naming
// the site. Without the macro the checks compile to nothing.
#ifdef ASC_SELF_CHECK
__device__ unsigned long long g_self_check;
__device__ __noinline__ bool self_check_fail(uint32_t site, uint64_t idx) {
    atomicCAS(&g_self_check, 0ull, ((unsigned long long)site << 32) | (idx & 0xffffffffull));
    return true;
}
#define ASC_BAD(cond, site, idx) ((cond) ? self_check_fail((site), (idx)) : false)
#else
#define ASC_BAD(cond, site, idx) false
#endif

enum Alg { kBFS = 0, kSSSP = 1, kCC = 2 };

// Control block (u32 words). Per parity p: [8p+0..3] counts of the frontier
// built for that parity (static list, on-demand list, static segments,
// on-demand segments), [8p+4..5] work cursors of the launches that build it,
// [8p+6..7] vertices of each region in that frontier (its bitmap's bits).
// Stats at word 16 (u64): edges static, edges on-demand, frontier vertices
// static, frontier vertices on-demand, reached vertices, reached edges. PageRank FP64 accumulators at word 32:
// residual[2], dangling[2].
// Word 28 counts iterations and word 29 flags an iteration cap hit when the
// loop runs on the device. Word 31 is the SSSP near-far threshold, words 36-39
// the minimum far distance of a pass.
// Words 42-43 (u64): in-edges that bottom-up BFS steps read from host memory;
// words 44-45 (u64): unreached vertices those steps examined. Words 46-47 (u64):
// in-edges of the vertices that a reference PageRank pass left active; words
// 48-55: vertices that a near-far promotion moved (two regions, four slots);
// 48-59: three residual and dangling-mass pairs (FP64) of PageRank passes, word
// 60 the ticket of the blocks that end a pass. Word 61 counts the arrivals at a
// grid barrier; word 29 is 2 when one ran out of time.
enum { CTL_BLOCK = 8, CTL_STATS = 16, CTL_ITERS = 28, CTL_TIMEOUT = 29, CTL_THRESH = 31,
       CTL_PR = 32, CTL_MINFAR = 36, CTL_BU_EDGES = 42, CTL_BU_VERTS = 44, CTL_ACTIVE = 46, CTL_PROMOTED = 48, CTL_ACC = 48,
       CTL_TICKET = 60, CTL_BARRIER = 61, CTL_WORDS = 64 };

struct RegionArgs {
    const uint32_t *ptr;
    const uint32_t *edges;        // region edge base, indexed by global edge offset
    uint32_t *val;
    uint32_t *bitmap;             // next-frontier bitmap (written)
    uint32_t *visited;            // BFS: reached-vertex bitmap (claims)
    const uint32_t *huge_bits;    // one bit per vertex whose list is cut into segments
    uint32_t *far_bits;           // SSSP near-far: vertices whose distance is at or above *thresh
    const uint32_t *thresh;
    const uint32_t *bitmap_in;    // this iteration's frontier bitmap (null: no id-order mode)
    const uint32_t *q_in;         // this region's input list (null: dense range)
    const uint64_t *seg_in;       // this region's input segments
    const uint32_t *cnt_in;       // counts of the input frontier
    uint32_t region;              // 0 static, 1 on-demand
    uint32_t dense_begin, dense_end;
    uint32_t *q_out;              // output lists: static at 0, on-demand at S
    uint64_t *seg_out;            // output segments: static at 0, on-demand at segcap_static
    uint32_t *cnt_out;
    uint32_t *work;
    unsigned long long *stats;
    uint32_t S;
    uint32_t huge;
    uint32_t seg_len;
    uint32_t segcap_static;
    uint32_t segcap_ondemand;
    uint32_t V;
    uint32_t dense_div;
    uint32_t wbits;               // > 0: u32 edges packed as (dst << wbits) | weight
    uint32_t ebits;               // bits per stored edge word: 32, or a bit stream of ebits per edge
    uint32_t item_div;            // by items while more than 1 / item_div of the region is active
    unsigned long long *frag;     // non-null: add edges read per 4096-edge fragment
    // bottom-up BFS steps (null in_ptr: top-down only)
    const uint32_t *in_ptr;       // in-edge offsets (device)
    const uint32_t *in_edges;     // in-edge source ids, a bit stream of in_ebits per edge (pinned host)
    uint32_t in_ebits;
    uint32_t bu_div;              // a step whose input frontier holds more than V / bu_div vertices is bottom-up
    uint32_t in_resident;         // in_edges is device memory (a graph without a cap), else pinned host
    const uint32_t *in_heads;     // first in-edge of every vertex in HBM (a bit stream of in_ebits), or null
    const uint32_t *in_none;      // one bit per vertex without in-edges (never reached but as a source)
    // merge items of the region (null: a region walked in id order is cut into
    // tiles of kBlock vertices and segments), and the words that may be read at edges
    const uint2 *items;
    uint32_t item_begin, item_n;
    uint64_t edge_words;
};

// True when this BFS iteration steps bottom-up: its input frontier (the
// region bit counts of the previous step, upper bounds) holds more than
// V / bu_div vertices. The top-down and bottom-up kernels of an iteration both
// evaluate it from the same counts and exactly one of them does the work.
__device__ __forceinline__ bool bottom_up_step(const RegionArgs &a, const uint32_t *cnt) {
    return a.in_ptr && a.bu_div && ((uint64_t)cnt[6] + cnt[7]) * a.bu_div > a.V;
}

// Adds the n edges read from [b, b + n) to their 4096-edge fragments' counters.
__device__ __forceinline__ void count_fragments(unsigned long long *frag, uint64_t b, uint32_t n) {
    if (!n) return;
    const uint64_t e = b + n;
    for (uint64_t f = b >> 12; f <= (e - 1) >> 12; f++) {
        const uint64_t lo = max(b, f << 12), hi = min(e, (f + 1) << 12);
        atomicAdd(frag + f, (unsigned long long)(hi - lo));
    }
}

// Edge layouts of the expansion kernels (their WORDS template argument):
// 1 = one u32 per edge, 2 = {dst, weight} pairs, kBitsLayout = one word per
// edge stored as a bit stream of ebits per edge.
constexpr int kBitsLayout = 3;

// ebits bits of a bit stream: edge idx at bits [idx*ebits, (idx+1)*ebits),
// little-endian across words; the buffer carries a padding word, so p[1]
// stays inside it.
__device__ __forceinline__ uint32_t bit_stream_word(const uint32_t *base, uint64_t idx, uint32_t ebits) {
    const uint64_t bit = idx * ebits;
    const uint32_t *p = base + (bit >> 5);
    const uint32_t sh = (uint32_t)bit & 31u;
    uint32_t x = __ldg(p) >> sh;
    if (sh + ebits > 32) x |= __ldg(p + 1) << (32 - sh);
    return x & ((1u << ebits) - 1u);
}

template <int WORDS>
__device__ __forceinline__ uint32_t layout_word(const uint32_t *base, uint64_t idx, uint32_t ebits) {
    return WORDS == kBitsLayout ? bit_stream_word(base, idx, ebits) : __ldg(base + idx);
}

// Edge word idx of a one-word-per-edge array: a plain load, or a bit-stream
// read when ebits < 32 (kernels with the layout as a template argument call
// bit_stream_word directly, without the per-edge test).
__device__ __forceinline__ uint32_t edge_word(const uint32_t *base, uint64_t idx, uint32_t ebits) {
    if (ebits == 32) return __ldg(base + idx);
    const uint64_t bit = idx * ebits;
    const uint32_t *p = base + (bit >> 5);
    const uint32_t sh = (uint32_t)bit & 31u;
    uint32_t x = __ldg(p) >> sh;
    if (sh + ebits > 32) x |= __ldg(p + 1) << (32 - sh);
    return x & ((1u << ebits) - 1u);
}

struct Smem {
    uint32_t pref[kBlock + 1];
    uint32_t start[kBlock];
    uint32_t vu[kBlock];
    uint32_t warp[kWarps + 1];
    uint32_t work;
};

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t &total, uint32_t *s_warp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t y = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        uint32_t t = lane < kWarps ? s_warp[lane] : 0;
        uint32_t ti = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            uint32_t y = __shfl_up_sync(kFull, ti, d);
            if (lane >= d) ti += y;
        }
        if (lane < kWarps) s_warp[lane] = ti - t;
        if (lane == kWarps - 1) s_warp[kWarps] = ti;
    }
    __syncthreads();
    total = s_warp[kWarps];
    return s_warp[w] + incl - x;
}

// Whether a region walked in id order goes by merge items or by tiles. Items hold
// equal work whatever the degrees; one with few active rows costs nearly as much to
// set up as a full one, a tile only its active edges, but a tile of kBlock vertices
// holds more edges than an item where degrees are high. So where the tiles of a graph
// are even (see kEvenTiles), items are for frontiers of over a quarter of the region
// at 8 edges per vertex and above, of over a sixteenth from 3 on, and for every dense
// frontier below. The on-demand region always goes by items, whose 16-byte reads keep
// the link's runs long where active vertices lie together (CC of 1 M vertices linked
// to 16 within 1,000 ids, 25% resident: 37.6 ms, by the rule 56.0). us, items for every
// dense frontier / above 1/16 / 1/8 / 1/4 / 1/2:
//   uniform random, 6 M vertices of 16: SSSP 6265 / 5715 / 5185 / 4808 / 4691
//   2 M of 8: SSSP 1468 / 1417 / 1384 / 1377 / 1375; of 4: 1067 / 1075 / 1077 / 1128 / 1151
//   of 2: 1073 / 1141 / 1205 / 1316 / 1313; grid of 1000 x 1000: 30420 / 29239 / 28998 /
//   28982 / 28986; RMAT scale 20 (uneven): CC 331 / 388 / 392 / 390 / 416
__device__ __forceinline__ bool by_items(const RegionArgs &a, uint32_t region, uint32_t bits, uint32_t range) {
    return a.items && (region || (uint64_t)bits * a.item_div > range);
}

// Merge items: a region's rows (each counted at its end) and edges in their
// merged order, cut every kItem positions. An item is the rows that end in it
// and the edges at its positions, so items hold equal work whatever the
// degrees; long lists span several. Passes and iterations that read most of a
// region run over its items, a CTA per item and kVt consecutive edges per thread.
// Both ways measured on the second iteration of a symmetrised RMAT graph of 6 M
// vertices (180 M edges, 355 MB of them over the host link): tiles of 256
// vertices, an owner search per edge and 4-byte reads 2.22 ms (160 GB/s over the
// link), items 1.77 (200 of the 211 a copy reaches).
constexpr int kVt = 8;
constexpr uint32_t kItem = kBlock * kVt;

// First (row, edge) of every item; items[n] is the end. Region 0 is the rows
// [0, S), region 1 the rows [S, V); each starts at an item boundary.
__global__ void merge_plan_kernel(const uint32_t *ptr, uint32_t S, uint32_t V, uint32_t L, uint32_t n0, uint32_t n,
                               uint2 *items) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        if (i == n) {
            items[i] = make_uint2(V, ptr[V]);
            continue;
        }
        const uint32_t R0 = i < n0 ? 0 : S, R1 = i < n0 ? S : V;
        const uint32_t E0 = ptr[R0];
        const uint64_t d = (uint64_t)(i - (i < n0 ? 0 : n0)) * L;
        // row r ends at merge position (its end - E0) + (r - R0): rows ending before d
        uint32_t lo = 0, hi = R1 - R0;
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if ((uint64_t)(ptr[R0 + mid + 1] - E0) + mid < d) lo = mid + 1;
            else hi = mid;
        }
        items[i] = make_uint2(R0 + lo, E0 + (uint32_t)(d - lo));
    }
}

// Words [w, w + 4) of an edge array of edge_words words, w a multiple of 4.
__device__ __forceinline__ uint4 load_words16(const uint32_t *edges, uint64_t edge_words, uint64_t w) {
    if (w + 4 <= edge_words) return __ldg(reinterpret_cast<const uint4 *>(edges + w));
    uint4 q;  // the buffer's last words
    q.x = w < edge_words ? __ldg(edges + w) : 0u;
    q.y = w + 1 < edge_words ? __ldg(edges + w + 1) : 0u;
    q.z = w + 2 < edge_words ? __ldg(edges + w + 2) : 0u;
    q.w = 0u;
    return q;
}

// Copies the words holding edges [e0, e0 + ne) to smem with 16-byte loads (so
// the host link serves runs of several KB); returns the bit of edge e0 there.
__device__ __forceinline__ uint32_t stage_words(const uint32_t *edges, uint64_t edge_words, uint32_t e0, uint32_t ne, uint32_t eb,
                                                   uint32_t *pool, uint32_t &nq) {
    const uint64_t bit = (uint64_t)e0 * eb;
    const uint64_t w_lo = (bit >> 5) & ~3ull;
    nq = ne ? (uint32_t)(((((uint64_t)e0 + ne) * eb + 31) / 32 - w_lo + 3) >> 2) : 0;
    for (uint32_t i = threadIdx.x; i < nq; i += kBlock)
        reinterpret_cast<uint4 *>(pool)[i] = load_words16(edges, edge_words, w_lo + 4ull * i);
    return (uint32_t)(bit - 32 * w_lo);
}

__device__ __forceinline__ uint32_t staged_word(const uint32_t *pool, uint32_t bit, uint32_t mask) {
    return __funnelshift_r(pool[bit >> 5], pool[(bit >> 5) + 1], bit & 31u) & mask;
}

template <int ALG, int WORDS>
__device__ __forceinline__ void load_edge(const RegionArgs &a, uint32_t vu, uint64_t idx, uint32_t &v, uint32_t &nv) {
    if (WORDS == 2) {
        uint2 e = __ldg(reinterpret_cast<const uint2 *>(a.edges) + idx);
        v = e.x;
        nv = ALG == kSSSP ? vu + e.y : (ALG == kBFS ? vu + 1 : vu);
    } else {
        const uint32_t e = layout_word<WORDS>(a.edges, idx, a.ebits);
        v = e >> a.wbits;
        nv = ALG == kBFS ? vu + 1 : (ALG == kSSSP ? vu + (e & ((1u << a.wbits) - 1u)) : vu);
    }
}

// Counts, per region, the vertices whose next-frontier bit this warp won
// (shared-memory counters, flushed once per CTA). Every lane calls it.
__device__ __forceinline__ void count_next(const RegionArgs &a, bool won, uint32_t v, uint32_t *s_next) {
    const unsigned m0 = __ballot_sync(kFull, won && v < a.S);
    const unsigned m1 = __ballot_sync(kFull, won && v >= a.S);
    if ((threadIdx.x & 31) == 0) {
        if (m0) atomicAdd(&s_next[0], (uint32_t)__popc(m0));
        if (m1) atomicAdd(&s_next[1], (uint32_t)__popc(m1));
    }
}

template <int ALG>
__device__ __forceinline__ uint32_t probe(const RegionArgs &a, uint32_t v) {
    return ALG == kBFS ? a.visited[v >> 5] : a.val[v];
}

#ifndef ASC_CLAIM_RED
#define ASC_CLAIM_RED 1
#endif
// Lowers val[v] to nv; true when this thread counts v into the next frontier.
// cur is the earlier probe: reached bits and values only ever grow / shrink,
// so a stale probe can only cost an extra atomic, never a missed update.
// BFS is level-synchronous: every update of an iteration writes the same
// level, so a thread whose probe found v unreached stores it and no atomicMin
// is needed (the result equals the atomicMin relaxation's fixpoint).
// With kClaimRed the atomics are fire-and-forget (no thread waits for a
// returned old value): two threads with stale probes may both store v's level
// (the same value) and both count v, so the per-region next-frontier counts
// are upper bounds. They only choose between list and bitmap walks and stop
// the loop when zero, which stays exact: a count is zero only when no thread
// set a bit. Otherwise the returned old bit decides, and counts are exact.
constexpr bool kClaimRed = ASC_CLAIM_RED != 0;
template <int ALG>
__device__ __forceinline__ bool lower(const RegionArgs &a, uint32_t v, uint32_t nv, uint32_t cur, uint32_t thresh) {
    const uint32_t bit = 1u << (v & 31);
    if (ALG == kBFS) {
        if (nv == 0xffffffffu || (cur & bit)) return false;
        if (kClaimRed) atomicOr(&a.visited[v >> 5], bit);
        else if (atomicOr(&a.visited[v >> 5], bit) & bit) return false;
        a.val[v] = nv;
        atomicOr(&a.bitmap[v >> 5], bit);
        return true;
    }
    if (nv >= cur) return false;
    if (ALG == kSSSP && a.far_bits) {
        // fire-and-forget, as below: a vertex lowered below the threshold by
        // another thread meanwhile may stay in the far set and is then expanded
        // once more when it is promoted
        atomicMin(&a.val[v], nv);
        if (nv >= thresh) {
            atomicOr(&a.far_bits[v >> 5], bit);  // waits until the threshold reaches it
            return false;
        }
        // now near: drop it from the far set, or a later promotion expands it twice
        if (a.far_bits[v >> 5] & bit) atomicAnd(&a.far_bits[v >> 5], ~bit);
    } else {
        // fire-and-forget: if another thread lowered v further since the probe,
        // it set v's bit too, so the next frontier is the same either way
        atomicMin(&a.val[v], nv);
    }
    if (kClaimRed) {
        atomicOr(&a.bitmap[v >> 5], bit);
        return true;
    }
    return (atomicOr(&a.bitmap[v >> 5], bit) & bit) == 0;
}

// Each thread handles kUnroll edges per pass: all column loads are issued
// first, then all destination-value loads, then the updates, so a thread keeps
// kUnroll independent reads in flight (on-demand column reads cross the host link).
// (measured with bit-packed edges at 8 CTAs per SM: 4 -> 65.7 GTEPS, 6 -> 64.3,
// 8 -> 62.2; more loads per thread spill at 32 registers)
#ifndef ASC_EXPAND_UNROLL
#define ASC_EXPAND_UNROLL 4
#endif
constexpr int kUnroll = ASC_EXPAND_UNROLL;

// Expands up to kBlock frontier vertices, one per thread (act = false where a
// thread has none): a block scan of their degrees lays the edges out as one
// range, which all threads walk kUnroll edges at a time.
template <int ALG, int WORDS>
__device__ void expand_vertices(const RegionArgs &a, bool act, uint32_t u, Smem &sm, uint32_t *s_next,
                                uint32_t thresh) {
    uint32_t deg = 0, start = 0, vu = 0;
    if (act && ASC_BAD(u >= a.V, 1, u)) act = false;
    if (act) {
        start = a.ptr[u];
        deg = a.ptr[u + 1] - start;
        if (deg > a.huge) {
            deg = 0;  // long lists are handled as segments
            act = false;
        }
        vu = a.val[u];
        if (a.frag) count_fragments(a.frag, start, deg);
    }
    uint32_t total;
    uint32_t excl = block_excl_scan(deg, total, sm.warp);
    sm.pref[threadIdx.x] = excl;
    sm.start[threadIdx.x] = start;
    sm.vu[threadIdx.x] = vu;
    if (threadIdx.x == 0) sm.pref[kBlock] = total;
    const uint32_t nact = __syncthreads_count(act);
    // each pass issues kUnroll column loads per thread before any update
    auto load_pass = [&](uint32_t base, uint32_t (&v)[kUnroll], uint32_t (&nv)[kUnroll]) {
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const uint32_t e = base + k * kBlock + threadIdx.x;
            v[k] = 0;
            nv[k] = 0xffffffffu;  // never lower than a value: no update
            if (e < total) {
                int lo = 0, hi = kBlock;
                while (hi - lo > 1) {
                    int mid = (lo + hi) >> 1;
                    if (sm.pref[mid] <= e) lo = mid;
                    else hi = mid;
                }
                load_edge<ALG, WORDS>(a, sm.vu[lo], (uint64_t)sm.start[lo] + (e - sm.pref[lo]), v[k], nv[k]);
                if (ASC_BAD(v[k] >= a.V, 2, v[k])) {
                    v[k] = 0;
                    nv[k] = 0xffffffffu;
                }
            }
        }
    };
    for (uint32_t base = 0; base < total; base += kUnroll * kBlock) {
        uint32_t v[kUnroll], nv[kUnroll], cur[kUnroll];
        load_pass(base, v, nv);
#pragma unroll
        for (int k = 0; k < kUnroll; k++) cur[k] = nv[k] != 0xffffffffu ? probe<ALG>(a, v[k]) : 0;
#pragma unroll
        for (int k = 0; k < kUnroll; k++) count_next(a, lower<ALG>(a, v[k], nv[k], cur[k], thresh), v[k], s_next);
    }
    if (threadIdx.x == 0) {
        atomicAdd(&a.stats[a.region], (unsigned long long)total);
        atomicAdd(&a.stats[2 + a.region], (unsigned long long)nact);
    }
    __syncthreads();
}

// One bitmap word of a region walked through its bitmap, bits outside
// [dense_begin, dense_end) cleared (u0 is 32-aligned).
__device__ __forceinline__ uint32_t region_word(const RegionArgs &a, uint32_t u0) {
    if (u0 >= a.dense_end) return 0u;
    uint32_t word = a.bitmap_in[u0 >> 5];
    if (u0 < a.dense_begin) word &= 0xffffffffu << (a.dense_begin - u0);
    if (a.dense_end - u0 < 32u) word &= (1u << (a.dense_end - u0)) - 1u;
    return word;
}

// One tile of frontier vertices, one per thread: per consecutive entries
// of the region's list, or (bitmap) kBlock consecutive vertex ids walked
// through the frontier bitmap (tiles start 32-aligned; a tile with no active
// vertex costs one bitmap read per warp).
template <int ALG, int WORDS>
__device__ __forceinline__ void expand_tile(const RegionArgs &a, uint32_t tile, uint32_t n_in, bool bitmap,
                                            uint32_t per, Smem &sm, uint32_t *s_next, uint32_t thresh) {
    bool act;
    uint32_t u;
    if (bitmap) {
        u = (a.dense_begin & ~31u) + tile * kBlock + threadIdx.x;
        act = (region_word(a, u & ~31u) >> (u & 31)) & 1u;
        if (!__syncthreads_or(act)) return;
    } else {
        const uint32_t i = tile * per + threadIdx.x;
        act = threadIdx.x < per && i < n_in;
        u = act ? a.q_in[i] : 0;
    }
    expand_vertices<ALG, WORDS>(a, act, u, sm, s_next, thresh);
}

template <int ALG, int WORDS>
__device__ void expand_segment(const RegionArgs &a, uint64_t item, uint32_t *s_next, uint32_t thresh) {
    const uint32_t u = (uint32_t)(item >> 32), k0 = (uint32_t)item;
    if (ASC_BAD(u >= a.V, 3, u)) return;
    const uint32_t b0 = a.ptr[u], e0 = a.ptr[u + 1];
    const uint64_t b = (uint64_t)b0 + (uint64_t)k0 * a.seg_len;
    const uint64_t e = min((uint64_t)e0, b + a.seg_len);
    const uint32_t n = (uint32_t)(e - b);
    const uint32_t vu = a.val[u];
    auto load_pass = [&](uint32_t base, uint32_t (&v)[kUnroll], uint32_t (&nv)[kUnroll]) {
#pragma unroll
        for (int k = 0; k < kUnroll; k++) {
            const uint32_t j = base + k * kBlock + threadIdx.x;
            v[k] = 0;
            nv[k] = 0xffffffffu;
            if (j < n) load_edge<ALG, WORDS>(a, vu, b + j, v[k], nv[k]);
            if (j < n && ASC_BAD(v[k] >= a.V, 2, v[k])) {
                v[k] = 0;
                nv[k] = 0xffffffffu;
            }
        }
    };
    for (uint32_t base = 0; base < n; base += kUnroll * kBlock) {
        uint32_t v[kUnroll], nv[kUnroll], cur[kUnroll];
        load_pass(base, v, nv);
#pragma unroll
        for (int k = 0; k < kUnroll; k++) cur[k] = nv[k] != 0xffffffffu ? probe<ALG>(a, v[k]) : 0;
#pragma unroll
        for (int k = 0; k < kUnroll; k++) count_next(a, lower<ALG>(a, v[k], nv[k], cur[k], thresh), v[k], s_next);
    }
    if (threadIdx.x == 0) {
        atomicAdd(&a.stats[a.region], (unsigned long long)n);
        if (k0 == 0) atomicAdd(&a.stats[2 + a.region], 1ull);
        if (a.frag) count_fragments(a.frag, b, n);
    }
}

// Work of one region for the bitmap-built frontier: segments first, then a
// region whose frontier holds more than 1/dense_div of its vertices is walked
// in id order through its bitmap (its list was not built), kBlock ids per
// item, so the lists of neighbouring active vertices are read as one
// contiguous run; otherwise through its list, per entries per item: as few as
// give every CTA of the grid one, at least kMinTile, since the lists of a tile
// are walked by one CTA (the third iteration of a BFS on RMAT scale 16 took 93
// us with its 800 vertices and 118,000 edges in four tiles of 256). An id-order walk
// by merge items (by_items) has no other items.
#ifndef ASC_MIN_TILE
#define ASC_MIN_TILE 8
#endif
constexpr uint32_t kMinTile = ASC_MIN_TILE;
// cnt: the frontier's counts (a.cnt_in or a copy). per is 0 for merge items.
__device__ __forceinline__ void region_items_bits(const RegionArgs &a, const uint32_t *cnt, uint32_t &n_in,
                                                  uint32_t &nseg, uint32_t &items, bool &bitmap, uint32_t &per) {
    const uint32_t range = a.dense_end - a.dense_begin;
    const uint32_t bits = cnt[6 + a.region];
    nseg = cnt[2 + a.region];
    bitmap = a.bitmap_in && a.dense_div && bits > range / a.dense_div;
    n_in = bitmap ? 0 : cnt[a.region];
    const uint32_t nvert = bitmap ? a.dense_end - (a.dense_begin & ~31u) : n_in;
    per = bitmap ? kBlock : min((uint32_t)kBlock, max(kMinTile, (n_in + gridDim.x - 1) / gridDim.x));
    items = nseg + (nvert + per - 1) / per;
    if (bitmap && by_items(a, a.region, bits, range)) {
        per = nseg = 0;
        items = a.item_n;
    }
}

// A region's merge item: the edges of its active rows, staged in shared memory
// by 16-byte chunks that hold any (so the host link serves long runs and only
// what is active), then kVt consecutive edges per thread. Val is what an active
// row carries to its edges.
template <int WORDS, typename Val>
struct ItemSmem {
    // the staged words, then one Val per row: at most ne (2 ne) words and nr + 1
    // Vals with nr + ne <= kItem, plus alignment and one word read past the end
    alignas(16) uint32_t pool[(WORDS == 2 || sizeof(Val) == 8 ? 2 : 1) * kItem + 24];
    uint16_t row_at[kItem];         // of an active row's first edge here: the row, from the item's first
    uint32_t starts[kItem / 32];    // one bit per edge: an active row starts here
    uint32_t active[kItem / 32];    // one bit per edge: it belongs to an active row
};

// The row of the last start before edge xw (a multiple of 32), when there is
// one. The whole warp calls it.
__device__ __forceinline__ uint32_t row_before(const uint32_t *starts, const uint16_t *row_at, uint32_t xw) {
    const int lane = threadIdx.x & 31;
    for (int m0 = (int)(xw >> 5) - 32; m0 > -32; m0 -= 32) {
        const uint32_t word = m0 + lane >= 0 ? starts[m0 + lane] : 0u;
        const unsigned any = __ballot_sync(kFull, word != 0);
        if (any) {
            const int q = 31 - __clz((int)any);
            const uint32_t bits = __shfl_sync(kFull, word, q);
            return row_at[32 * (m0 + q) + 31 - __clz((int)bits)];
        }
    }
    return 0;
}

// Stages item it; false when it holds no active edge. loads(u) is row u's Val;
// counts (shared) receive the edges and vertices. The block calls it together.
template <int WORDS, typename Val, typename Load>
__device__ __forceinline__ bool stage_merge_item(const RegionArgs &a, uint32_t it, ItemSmem<WORDS, Val> &sm, Load load,
                                                 uint32_t *n_edges, uint32_t *n_verts, uint32_t &ne_out,
                                                 uint32_t &bit0_out, Val *&value) {
    const uint2 i0 = a.items[it], i1 = a.items[it + 1];
    const uint32_t r0 = i0.x, e0 = i0.y, nr = i1.x - i0.x, ne = i1.y - i0.y;
    const int lane = threadIdx.x & 31;
    const uint32_t eb = WORDS == 2 ? 64 : WORDS == 1 ? 32 : a.ebits;
    const uint64_t bit = (uint64_t)e0 * eb, w_lo = (bit >> 5) & ~3ull;
    const uint32_t bit0 = (uint32_t)(bit - 32 * w_lo), nq = (bit0 + ne * eb + 127) >> 7;
    value = reinterpret_cast<Val *>(sm.pool + 4 * nq + 4);
    ne_out = ne;
    bit0_out = bit0;
    if (threadIdx.x < kItem / 32) sm.starts[threadIdx.x] = sm.active[threadIdx.x] = 0;
    __syncthreads();
    uint32_t edges = 0, verts = 0;
    for (uint32_t j = threadIdx.x; j <= nr; j += kBlock) {
        const uint32_t u = r0 + j;
        if (u >= a.dense_end || !((a.bitmap_in[u >> 5] >> (u & 31)) & 1u)) continue;
        const uint32_t b = a.ptr[u], e = a.ptr[u + 1];
        const uint32_t lo = b > e0 ? b - e0 : 0, hi = min(e - e0, ne);
        verts += j < nr;  // a vertex counts where its row ends
        if (lo >= hi) continue;
        edges += hi - lo;
        value[j] = load(u);
        sm.row_at[lo] = (uint16_t)j;
        atomicOr(&sm.starts[lo >> 5], 1u << (lo & 31));
        for (uint32_t w = lo >> 5; w <= (hi - 1) >> 5; w++) {
            uint32_t m = 0xffffffffu;
            if (w == lo >> 5) m &= 0xffffffffu << (lo & 31);
            if (w == (hi - 1) >> 5) m &= 0xffffffffu >> (31 - ((hi - 1) & 31));
            atomicOr(&sm.active[w], m);
        }
        if (a.frag) count_fragments(a.frag, (uint64_t)e0 + lo, hi - lo);
    }
    const bool any = __syncthreads_or(edges != 0);
    edges = __reduce_add_sync(kFull, edges);
    verts = __reduce_add_sync(kFull, verts);
    if (lane == 0 && edges) atomicAdd(n_edges, edges);
    if (lane == 0 && verts) atomicAdd(n_verts, verts);
    if (!any) return false;
    for (uint32_t i = threadIdx.x; i < nq; i += kBlock) {
        // edges with a bit in this chunk
        const uint32_t c0 = 128 * i;
        const uint32_t x0 = c0 > bit0 ? (c0 - bit0) / eb : 0, x1 = min(ne - 1, (c0 + 127 - bit0) / eb);
        uint32_t need = 0;
        for (uint32_t w = x0 >> 5; w <= x1 >> 5; w++) {
            uint32_t m = sm.active[w];
            if (w == x0 >> 5) m &= 0xffffffffu << (x0 & 31);
            if (w == x1 >> 5) m &= 0xffffffffu >> (31 - (x1 & 31));
            need |= m;
        }
        if (need) reinterpret_cast<uint4 *>(sm.pool)[i] = load_words16(a.edges, a.edge_words, w_lo + 4ull * i);
    }
    __syncthreads();
    return true;
}

// A thread's kVt edges of a staged item: which are active, where rows start, and
// the Val of the row open at the first one (when that is active). False for the
// whole warp when it has none.
template <int WORDS, typename Val>
__device__ __forceinline__ bool merge_item_edges(const ItemSmem<WORDS, Val> &sm, const Val *value, uint32_t ne,
                                                 uint32_t x0, uint32_t &act, uint32_t &st, Val &open) {
    const int lane = threadIdx.x & 31;
    const uint32_t xw = x0 - lane * kVt;  // the warp's first edge
    if (xw >= ne) return false;
    act = (sm.active[x0 >> 5] >> (x0 & 31)) & ((1u << kVt) - 1u);
    st = (sm.starts[x0 >> 5] >> (x0 & 31)) & ((1u << kVt) - 1u);
    if (!__any_sync(kFull, act != 0)) return false;
    // of the last start in an earlier lane, or in an earlier warp
    const unsigned began = __ballot_sync(kFull, st != 0);
    const uint32_t last = st ? sm.row_at[x0 + 31 - __clz((int)st)] : 0u;
    const unsigned below = began & ((1u << lane) - 1u);
    const uint32_t from_lane = __shfl_sync(kFull, last, below ? 31 - __clz((int)below) : lane);
    const uint32_t before = row_before(sm.starts, sm.row_at, xw);
    const uint32_t row = (st & 1u) ? (uint32_t)sm.row_at[x0] : below ? from_lane : before;
    open = (act & 1u) ? value[row] : (Val)0;
    return true;
}

template <int ALG, int WORDS>
__device__ void expand_merge_item(const RegionArgs &a, uint32_t it, ItemSmem<WORDS, uint32_t> &sm, uint32_t *s_next,
                                  uint32_t thresh) {
    uint32_t ne, bit0, *value;
    if (!stage_merge_item(a, it, sm, [&](uint32_t u) { return a.val[u]; }, &s_next[2 + a.region],
                          &s_next[4 + a.region], ne, bit0, value))
        return;
    const uint32_t eb = WORDS == 2 ? 64 : WORDS == 1 ? 32 : a.ebits;
    const uint32_t mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
    const uint32_t x0 = threadIdx.x * kVt;
    uint32_t n0 = 0, n1 = 0, act, st, vu;
    if (merge_item_edges(sm, value, ne, x0, act, st, vu)) {
#pragma unroll
        for (int k0 = 0; k0 < kVt; k0 += kUnroll) {
            uint32_t v[kUnroll], nv[kUnroll], cur[kUnroll];
#pragma unroll
            for (int k = 0; k < kUnroll; k++) {
                v[k] = 0;
                nv[k] = 0xffffffffu;  // never lower than a value: no update
                if ((act >> (k0 + k)) & 1u) {
                    if (k0 + k > 0 && ((st >> (k0 + k)) & 1u)) vu = value[sm.row_at[x0 + k0 + k]];
                    const uint32_t at = bit0 + (x0 + k0 + k) * eb;
                    if (WORDS == 2) {
                        v[k] = sm.pool[at >> 5];
                        nv[k] = ALG == kSSSP ? vu + sm.pool[(at >> 5) + 1] : (ALG == kBFS ? vu + 1 : vu);
                    } else {
                        const uint32_t e = WORDS == 1 ? sm.pool[at >> 5] : staged_word(sm.pool, at, mask);
                        v[k] = e >> a.wbits;
                        nv[k] = ALG == kBFS ? vu + 1 : (ALG == kSSSP ? vu + (e & ((1u << a.wbits) - 1u)) : vu);
                    }
                    if (ASC_BAD(v[k] >= a.V, 2, v[k])) {
                        v[k] = 0;
                        nv[k] = 0xffffffffu;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kUnroll; k++) cur[k] = nv[k] != 0xffffffffu ? probe<ALG>(a, v[k]) : 0;
#pragma unroll
            for (int k = 0; k < kUnroll; k++) {
                const bool won = lower<ALG>(a, v[k], nv[k], cur[k], thresh);
                n0 += won && v[k] < a.S;
                n1 += won && v[k] >= a.S;
            }
        }
    }
    n0 = __reduce_add_sync(kFull, n0);
    n1 = __reduce_add_sync(kFull, n1);
    if ((threadIdx.x & 31) == 0 && n0) atomicAdd(&s_next[0], n0);
    if ((threadIdx.x & 31) == 0 && n1) atomicAdd(&s_next[1], n1);
    __syncthreads();
}

// Shared memory of an expansion: a tile's or a merge item's.
template <int WORDS>
union ExpandSmem {
    Smem tile;
    ItemSmem<WORDS, uint32_t> item;
};
// Shared counters of an expansion: next-frontier vertices per region, then the
// edges and the vertices that merge items expanded.
constexpr int kNextWords = 6;

template <int ALG, int WORDS>
__device__ __forceinline__ void expand_item(const RegionArgs &a, uint32_t w, uint32_t n_in, uint32_t nseg,
                                            bool bitmap, uint32_t per, ExpandSmem<WORDS> &sm, uint32_t *s_next,
                                            uint32_t thresh) {
    if (w < nseg) expand_segment<ALG, WORDS>(a, a.seg_in[w], s_next, thresh);
    else if (!per) expand_merge_item<ALG, WORDS>(a, a.item_begin + w, sm.item, s_next, thresh);
    else expand_tile<ALG, WORDS>(a, w - nseg, n_in, bitmap, per, sm.tile, s_next, thresh);
}

__device__ __forceinline__ void flush_next(const RegionArgs &a, uint32_t *s_next) {
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_next[0]) atomicAdd(&a.cnt_out[6], s_next[0]);
        if (s_next[1]) atomicAdd(&a.cnt_out[7], s_next[1]);
    }
}

// The same with what merge items counted.
__device__ __forceinline__ void flush_expansion(const RegionArgs &a, uint32_t *s_next) {
    flush_next(a, s_next);
    if (threadIdx.x < 4 && s_next[2 + threadIdx.x])
        atomicAdd(&a.stats[threadIdx.x], (unsigned long long)s_next[2 + threadIdx.x]);
}

template <int ALG, int WORDS>
__global__ void __launch_bounds__(kBlock, ASC_EXPAND_MIN_BLOCKS) expand_kernel(RegionArgs a) {
    if (ALG == kBFS && bottom_up_step(a, a.cnt_in)) return;
    __shared__ ExpandSmem<WORDS> sm;
    __shared__ uint32_t s_next[kNextWords], s_work;
    if (threadIdx.x < kNextWords) s_next[threadIdx.x] = 0;
    uint32_t n_in, nseg, total;
    bool bitmap;
    uint32_t per;
    region_items_bits(a, a.cnt_in, n_in, nseg, total, bitmap, per);
    const uint32_t thresh = ALG == kSSSP && a.far_bits ? *a.thresh : 0u;
    for (;;) {
        if (threadIdx.x == 0) s_work = atomicAdd(a.work, 1u);
        __syncthreads();
        const uint32_t w = s_work;
        __syncthreads();
        if (w >= total) break;
        expand_item<ALG, WORDS>(a, w, n_in, nseg, bitmap, per, sm, s_next, thresh);
    }
    flush_expansion(a, s_next);
}

// Both regions in one launch. Work items alternate between the on-demand and
// the static region while both have items left, so every SM mixes HBM-bound
// static work with link-bound on-demand work; on-demand segments and tiles
// are handed out first within their region.
struct FusedArgs {
    RegionArgs r0, r1;
    uint32_t *work;
};

// A CTA's first item is its own number; later ones come from the cursor, which
// starts behind them. cnt: the frontier's counts.
template <int ALG, int WORDS>
__device__ __forceinline__ void expand_regions(const FusedArgs &x, const uint32_t *cnt, uint32_t thresh,
                                               ExpandSmem<WORDS> &sm, uint32_t *s_next) {
    __shared__ uint32_t s_work;
    uint32_t n0, s0, i0, t0, n1, s1, i1, t1;
    bool m0, m1;
    region_items_bits(x.r0, cnt, n0, s0, i0, m0, t0);
    region_items_bits(x.r1, cnt, n1, s1, i1, m1, t1);
    const uint32_t m = min(i0, i1), total = i0 + i1;
    if (threadIdx.x < kNextWords) s_next[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t w = blockIdx.x; w < total;) {
        bool od;
        uint32_t local;
        if (w < 2 * m) {
            od = (w & 1) == 0;
            local = w >> 1;
        } else {
            od = i1 > i0;
            local = m + (w - 2 * m);
        }
        if (threadIdx.x == 0) s_work = gridDim.x + atomicAdd(x.work, 1u);
        if (od) expand_item<ALG, WORDS>(x.r1, local, n1, s1, m1, t1, sm, s_next, thresh);
        else expand_item<ALG, WORDS>(x.r0, local, n0, s0, m0, t0, sm, s_next, thresh);
        __syncthreads();
        w = s_work;
        __syncthreads();
    }
    flush_expansion(x.r0, s_next);
}

template <int ALG, int WORDS>
__global__ void __launch_bounds__(kBlock, ASC_EXPAND_MIN_BLOCKS) expand_fused_kernel(FusedArgs x) {
    if (ALG == kBFS && bottom_up_step(x.r0, x.r0.cnt_in)) return;
    __shared__ ExpandSmem<WORDS> sm;
    __shared__ uint32_t s_next[kNextWords];
    expand_regions<ALG, WORDS>(x, x.r0.cnt_in, ALG == kSSSP && x.r0.far_bits ? *x.r0.thresh : 0u, sm, s_next);
}

// Bottom-up BFS step (direction-optimizing BFS): every vertex not yet reached
// scans its in-edges, from the one whose source has the most out-edges on, for a
// parent in this iteration's frontier and stops at the first one; a vertex found
// takes the parent's value + 1 (the level-synchronous top-down step gives every
// unreached vertex with a frontier in-neighbour the same value, so levels are
// identical) and joins the next frontier. When the frontier is a large part of the graph, most unreached
// vertices find a parent among their first in-edges, so the step reads far
// fewer edge bytes over the host link than expanding the frontier's out-lists.
// A warp takes bitmap words of 32 vertices, lane = vertex, and writes the bits of
// those whose first in-edge is a parent; bits of vertices found later are added.
// Further in-edges are read in place from pinned host memory (device memory on a
// graph without a cap), kBuUnroll per lane before any frontier probe.
#ifndef ASC_BU_UNROLL
#define ASC_BU_UNROLL 4
#endif
constexpr int kBuUnroll = ASC_BU_UNROLL;

// Words a warp takes per pass: all of their bitmap words, heads and frontier
// probes are loaded before any is used, so a warp keeps that many independent
// load chains in flight.
#ifndef ASC_BU_WORDS
#define ASC_BU_WORDS 4
#endif
constexpr int kBuWords = ASC_BU_WORDS;
// CTAs per SM the bottom-up kernel is compiled for; its grid is one wave of
// them: at 8 it would spill (6 M vertices of 16 random neighbours, 25% resident,
// host-driven loop: 2.93 ms at 8, 2.73 at 6; RMAT scale 22: 0.652 and 0.655).
#ifndef ASC_BU_MIN_BLOCKS
#define ASC_BU_MIN_BLOCKS 6
#endif
constexpr int kBuMinBlocks = ASC_BU_MIN_BLOCKS;

// Vertices whose first in-edge is no parent scan the others: a chain of three
// dependent reads (in_ptr, then host memory). A word of 32 vertices with kBuDirect of
// them or more scans at once, as one run of lists; fewer wait in a queue per warp
// until 32 scan together (BFS on RMAT scale 24: 651 us a word at a time, 575 queued).
constexpr uint32_t kBuDirect = 24;
struct BuSmem {
    uint32_t queue[kWarps][32 + (kBuDirect - 1) * kBuWords];
    uint32_t open[kWarps][kBuWords];  // of a word that scans at once: its vertices
};

// Whether an in-edge of v after its first comes from the frontier, in the lanes that
// want to know. Lists in host memory are read 16 aligned bytes at a time: word by
// word, their sectors came over the link again and again, as often as the L1 had lost
// them meanwhile (2 M vertices of 16 random neighbours, 25% resident: 10.0 M sectors
// for 62 MB of lists, BFS 2.85 ms; 1.68 so). Resident lists come from L2, where that
// costs little and the fewer instructions count (500,009 vertices of a rewired ring,
// host-driven loop: 1.75 ms a word at a time, 1.91 by 16 bytes).
__device__ __forceinline__ bool bottom_up_scan(const RegionArgs &a, bool want, uint32_t v, uint32_t &scanned) {
    const uint32_t eb = a.in_ebits, mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
    uint32_t i = 0, e = 0;
    if (want) {
        i = a.in_ptr[v];
        e = a.in_ptr[v + 1];
        if (a.in_heads && i < e) i++;  // the head was the first
    }
    bool found = false;
    if (a.in_resident) {
        for (; i < e && !found; i += kBuUnroll) {
            uint32_t u[kBuUnroll];
            bool in[kBuUnroll];
#pragma unroll
            for (int k = 0; k < kBuUnroll; k++) {
                u[k] = i + k < e ? edge_word(a.in_edges, (uint64_t)i + k, eb) : 0xffffffffu;
                if (u[k] != 0xffffffffu && ASC_BAD(u[k] >= a.V, 17, u[k])) u[k] = 0xffffffffu;
            }
#pragma unroll
            for (int k = 0; k < kBuUnroll; k++)
                in[k] = u[k] != 0xffffffffu && ((a.bitmap_in[u[k] >> 5] >> (u[k] & 31)) & 1u);
            // edges read count up to the parent
#pragma unroll
            for (int k = 0; k < kBuUnroll; k++)
                if (!found && i + k < e) {
                    scanned++;
                    found = in[k];
                }
        }
        return found;
    }
    while (i < e && !found) {
        const uint64_t bit = (uint64_t)i * eb, w = (bit >> 5) & ~3ull;
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(a.in_edges + w));  // the array ends on 16 bytes
        // the last edge that begins in these words may end in the next one
        const uint32_t q4 = (uint64_t)e * eb > 32 * (w + 4) ? __ldg(a.in_edges + w + 4) : 0u;
        for (uint32_t at = (uint32_t)(bit - 32 * w); at < 128 && i < e && !found;) {
            uint32_t u[kBuUnroll], n = 0;
            bool in[kBuUnroll];
#pragma unroll
            for (int k = 0; k < kBuUnroll; k++) {
                const uint32_t x = at >> 5;
                const uint32_t lo = x == 0 ? q.x : x == 1 ? q.y : x == 2 ? q.z : q.w;
                const uint32_t hi = x == 0 ? q.y : x == 1 ? q.z : x == 2 ? q.w : q4;
                const bool begins = at < 128 && i + k < e;
                n += begins;
                u[k] = begins ? __funnelshift_r(lo, hi, at & 31u) & mask : 0xffffffffu;
                if (u[k] != 0xffffffffu && ASC_BAD(u[k] >= a.V, 17, u[k])) u[k] = 0xffffffffu;
                at += eb;
            }
#pragma unroll
            for (int k = 0; k < kBuUnroll; k++)
                in[k] = u[k] != 0xffffffffu && ((a.bitmap_in[u[k] >> 5] >> (u[k] & 31)) & 1u);
            // edges read count up to the parent
#pragma unroll
            for (int k = 0; k < kBuUnroll; k++)
                if (!found && u[k] != 0xffffffffu) {
                    scanned++;
                    found = in[k];
                }
            i += n;
        }
    }
    return found;
}

// nv: the value of a vertex found in this step (every frontier vertex holds
// nv - 1: the loop is level-synchronous).
__device__ __forceinline__ void bottom_up_words(const RegionArgs &a, uint32_t nwords, uint32_t nv, BuSmem &bs,
                                                uint32_t *s_next) {
    if (threadIdx.x < kNextWords) s_next[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * kWarps;
    uint32_t *queue = bs.queue[threadIdx.x >> 5];
    uint32_t waiting = 0, scanned = 0, examined = 0, n0 = 0, n1 = 0;
    // as many words a pass, up to kBuWords, as spread them evenly over the passes: with
    // kBuWords in each, 31,250 words of 1 M vertices took 7,296 warps through a second
    // pass for the last 516 (100 steps of a graph of 100 layers: 4.0 ms, 3.1 so)
    const uint32_t passes = (nwords - 1) / (kBuWords * warps) + 1;
    const uint32_t step = (nwords - 1) / (passes * warps) + 1;
    for (uint32_t w0 = step * (blockIdx.x * kWarps + (threadIdx.x >> 5)); w0 < nwords; w0 += step * warps) {
        // vertices without in-edges can never be reached: about half of an
        // RMAT graph, nearly all of its unreachable vertices
        uint32_t vis[kBuWords], done[kBuWords], dense = 0;
#pragma unroll
        for (int k = 0; k < kBuWords; k++) {
            const bool in = k < (int)step && w0 + k < nwords;
            vis[k] = in ? a.visited[w0 + k] : 0xffffffffu;
            done[k] = in ? vis[k] | a.in_none[w0 + k] : 0xffffffffu;
        }
        // the first in-edge is held in HBM, vertex-indexed (a coalesced read;
        // a vertex without in-edges holds its own id, never in the frontier):
        // most unreached vertices find their parent there and read nothing else
        uint32_t head[kBuWords];
        bool todo[kBuWords], hit[kBuWords];
#pragma unroll
        for (int k = 0; k < kBuWords; k++) {
            const uint32_t v = 32 * (w0 + k) + lane;
            todo[k] = done[k] != 0xffffffffu && v < a.V && !((done[k] >> lane) & 1u);
            head[k] = todo[k] && a.in_heads ? edge_word(a.in_heads, v, a.in_ebits) : 0u;
            if (ASC_BAD(head[k] >= a.V, 16, head[k])) head[k] = v;
        }
#pragma unroll
        for (int k = 0; k < kBuWords; k++)
            hit[k] = todo[k] && a.in_heads && ((a.bitmap_in[head[k] >> 5] >> (head[k] & 31)) & 1u);
#pragma unroll
        for (int k = 0; k < kBuWords; k++) {
            if (done[k] == 0xffffffffu) continue;  // the whole warp: nothing to look for in this word
            const uint32_t w = w0 + k, v = 32 * w + lane;
            examined += todo[k];
            const unsigned found = __ballot_sync(kFull, hit[k]);
            if (hit[k]) {
                a.val[v] = nv;
                n0 += v < a.S;
                n1 += v >= a.S;
            }
            if (lane == 0 && found) {
                a.visited[w] = vis[k] | found;
                a.bitmap[w] = found;
            }
            const bool miss = todo[k] && !hit[k];
            const unsigned missed = __ballot_sync(kFull, miss);
            if (__popc(missed) >= kBuDirect) {
                dense |= 1u << k;
                if (lane == 0) bs.open[threadIdx.x >> 5][k] = missed;
                continue;
            }
            if (miss) queue[waiting + __popc(missed & ((1u << lane) - 1u))] = v;
            waiting += __popc(missed);
        }
        __syncwarp();  // the queue, and these words' bits before later ones are added
        const bool last = w0 + step * warps >= nwords;
        while (dense || waiting >= 32 || (last && waiting)) {  // one scan for both: code is fetched too
            uint32_t v, w = 0xffffffffu;
            bool want;
            if (dense) {
                const int k = __ffs((int)dense) - 1;
                dense &= dense - 1;
                w = w0 + k;
                v = 32 * w + lane;
                want = (bs.open[threadIdx.x >> 5][k] >> lane) & 1u;
            } else {
                const uint32_t n = min(waiting, 32u);
                waiting -= n;
                want = lane < n;
                v = want ? queue[waiting + lane] : 0u;
            }
            const bool found = bottom_up_scan(a, want, v, scanned);
            const unsigned all = __ballot_sync(kFull, found);
            if (found) {
                a.val[v] = nv;
                n0 += v < a.S;
                n1 += v >= a.S;
                if (w == 0xffffffffu) {
                    atomicOr(&a.visited[v >> 5], 1u << (v & 31));
                    atomicOr(&a.bitmap[v >> 5], 1u << (v & 31));
                }
            }
            if (w != 0xffffffffu && lane == 0 && all) {
                atomicOr(&a.visited[w], all);
                atomicOr(&a.bitmap[w], all);
            }
            __syncwarp();
        }
    }
    n0 = __reduce_add_sync(kFull, n0);
    n1 = __reduce_add_sync(kFull, n1);
    scanned = __reduce_add_sync(kFull, scanned);
    examined = __reduce_add_sync(kFull, examined);
    if (lane == 0) {
        if (n0) atomicAdd(&s_next[0], n0);
        if (n1) atomicAdd(&s_next[1], n1);
        if (scanned) atomicAdd(&s_next[2], scanned);
        if (examined) atomicAdd(&s_next[3], examined);
    }
    flush_next(a, s_next);
    if (threadIdx.x == 0 && s_next[3])
        atomicAdd((unsigned long long *)(a.stats + (CTL_BU_VERTS - CTL_STATS) / 2), (unsigned long long)s_next[3]);
    // in-edges are read in place from host memory (resident only on a graph
    // without a cap): the run's on-demand edges and its bottom-up edges
    if (threadIdx.x == 0 && s_next[2]) {
        atomicAdd(&a.stats[a.in_resident ? 0 : 1], (unsigned long long)s_next[2]);
        atomicAdd((unsigned long long *)(a.stats + (CTL_BU_EDGES - CTL_STATS) / 2), (unsigned long long)s_next[2]);
    }
}

__global__ void __launch_bounds__(kBlock, kBuMinBlocks) bottom_up_kernel(RegionArgs a, uint32_t nwords, uint32_t nv) {
    if (!bottom_up_step(a, a.cnt_in)) return;
    __shared__ uint32_t s_next[kNextWords];
    __shared__ BuSmem bs;
    bottom_up_words(a, nwords, nv, bs, s_next);
}

// Gather-and-copy comparison engine: expands on-demand edges that host
// threads gathered into a device staging buffer. Item i is (vertex, offset of
// its edges in the staging buffer, edge count, 1 for a vertex's first item);
// a warp takes an item, its lanes 32 edges at a time. Staged edges are plain
// words (WORDS 1: destination or packed destination/weight) or pairs (2).
struct StagedArgs {
    RegionArgs a;
    const uint32_t *stage;
    const uint32_t *items;
    uint32_t n_items;
};

template <int ALG, int WORDS>
__global__ void __launch_bounds__(kBlock) expand_staged_kernel(StagedArgs x) {
    __shared__ uint32_t s_next[2];
    if (threadIdx.x < 2) s_next[threadIdx.x] = 0;
    __syncthreads();
    const RegionArgs &a = x.a;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = warp; i < x.n_items; i += nwarps) {
        const uint32_t u = x.items[4 * i], off = x.items[4 * i + 1], len = x.items[4 * i + 2];
        const uint32_t vu = a.val[u];
        for (uint32_t j0 = 0; j0 < len; j0 += 32) {
            const uint32_t j = j0 + lane;
            uint32_t v = 0, nv = 0xffffffffu;
            if (j < len) {
                if (WORDS == 2) {
                    const uint2 e = reinterpret_cast<const uint2 *>(x.stage)[(uint64_t)off + j];
                    v = e.x;
                    nv = ALG == kSSSP ? vu + e.y : (ALG == kBFS ? vu + 1 : vu);
                } else {
                    const uint32_t e = x.stage[(uint64_t)off + j];
                    v = e >> a.wbits;
                    nv = ALG == kBFS ? vu + 1 : (ALG == kSSSP ? vu + (e & ((1u << a.wbits) - 1u)) : vu);
                }
            }
            const uint32_t cur = nv != 0xffffffffu ? probe<ALG>(a, v) : 0;
            count_next(a, lower<ALG>(a, v, nv, cur, a.far_bits ? *a.thresh : 0u), v, s_next);
        }
        if (lane == 0) {
            atomicAdd(&a.stats[1], (unsigned long long)len);
            if (x.items[4 * i + 3]) atomicAdd(&a.stats[3], 1ull);
        }
    }
    flush_next(a, s_next);
}

// Builds the next frontier from its bitmap (one thread per 32-vertex word):
// vertices with long lists become segment items; the others are appended to
// their region's list only when that region will be walked as a list (warp
// scan of the per-word counts, one atomic per warp). bits0 and bits1 are the
// region bit counts (cnt_out[6..7], which the expansion flushed); cnt_out[0..3]
// receive the lists.
__device__ __forceinline__ void build_frontier(const RegionArgs &a, const uint32_t *next_bits, uint32_t nwords,
                                               uint32_t bits0, uint32_t bits1) {
    const int lane = threadIdx.x & 31;
    const uint32_t range0 = a.S, range1 = a.V - a.S;
    const bool list0 = !(a.dense_div && bits0 > range0 / a.dense_div);
    const bool list1 = !(a.dense_div && bits1 > range1 / a.dense_div);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < nwords; base += stride) {
        const uint32_t w = base + threadIdx.x;
        uint32_t word = 0, hw = 0;
        if (w < nwords) {
            word = next_bits[w];
            hw = word & a.huge_bits[w];
        }
        // region split of this word: bits of vertices below S are static
        uint32_t smask;
        const uint32_t v0 = 32 * w;
        if (v0 + 32 <= a.S) smask = 0xffffffffu;
        else if (v0 >= a.S) smask = 0;
        else smask = (1u << (a.S - v0)) - 1u;
        // long lists: one thread per vertex appends its segments (rare); merge
        // items need none
        if (!list0 && by_items(a, 0, bits0, range0)) hw &= ~smask;
        if (!list1 && by_items(a, 1, bits1, range1)) hw &= smask;
        while (hw) {
            const int b = __ffs(hw) - 1;
            hw &= hw - 1;
            const uint32_t v = 32 * w + b;
            const uint32_t deg = a.ptr[v + 1] - a.ptr[v];
            const uint32_t nseg = (deg + a.seg_len - 1) / a.seg_len;
            const bool od = v >= a.S;
            const uint32_t sb = atomicAdd(&a.cnt_out[2 + od], nseg);
            if (ASC_BAD((uint64_t)sb + nseg > (od ? a.segcap_ondemand : a.segcap_static), 13, sb)) continue;
            uint64_t *dst = a.seg_out + (od ? a.segcap_static : 0) + sb;
            for (uint32_t k = 0; k < nseg; k++) dst[k] = ((uint64_t)v << 32) | k;
        }
        if (w < nwords) word &= ~a.huge_bits[w];
        const uint32_t w0 = list0 ? (word & smask) : 0, w1 = list1 ? (word & ~smask) : 0;
        const uint32_t c0 = __popc(w0), c1 = __popc(w1);
        uint32_t i0 = c0, i1 = c1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y0 = __shfl_up_sync(kFull, i0, d), y1 = __shfl_up_sync(kFull, i1, d);
            if (lane >= d) {
                i0 += y0;
                i1 += y1;
            }
        }
        const uint32_t t0 = __shfl_sync(kFull, i0, 31), t1 = __shfl_sync(kFull, i1, 31);
        uint32_t b0 = 0, b1 = 0;
        if (lane == 0) {
            if (t0) b0 = atomicAdd(&a.cnt_out[0], t0);
            if (t1) b1 = atomicAdd(&a.cnt_out[1], t1);
        }
        b0 = __shfl_sync(kFull, b0, 0) + i0 - c0;
        b1 = __shfl_sync(kFull, b1, 0) + i1 - c1;
        uint32_t x = w0;
        while (x) {
            const int b = __ffs(x) - 1;
            x &= x - 1;
            if (!ASC_BAD(b0 >= a.S, 14, b0)) a.q_out[b0] = v0 + b;
            b0++;
        }
        x = w1;
        while (x) {
            const int b = __ffs(x) - 1;
            x &= x - 1;
            if (!ASC_BAD(a.S + b1 >= a.V, 15, b1)) a.q_out[a.S + b1] = v0 + b;
            b1++;
        }
    }
}

__global__ void build_frontier_kernel(RegionArgs a, const uint32_t *next_bits, uint32_t nwords) {
    build_frontier(a, next_bits, nwords, a.cnt_out[6], a.cnt_out[7]);
}

// SSSP near-far, step 1: when the pass left the near frontier empty, the
// smallest distance in the far set (atomicMin into the control block).
__global__ void far_min_kernel(RegionArgs a, uint32_t nwords, uint32_t *minfar) {
    if (a.cnt_out[6] | a.cnt_out[7]) return;
    uint32_t m = 0xffffffffu;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        uint32_t word = a.far_bits[w];
        while (word) {
            const int b = __ffs(word) - 1;
            word &= word - 1;
            m = min(m, a.val[32 * w + b]);
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = min(m, __shfl_down_sync(kFull, m, d));
    if ((threadIdx.x & 31) == 0 && m != 0xffffffffu) atomicMin(minfar, m);
}

// SSSP near-far, step 2: the threshold moves to (min far distance + delta) and
// every far vertex below it joins the next frontier (bit and region count).
__global__ void far_promote_kernel(RegionArgs a, uint32_t nwords, const uint32_t *minfar, uint32_t *thresh,
                                   uint32_t delta) {
    if (a.cnt_out[6] | a.cnt_out[7]) return;
    const uint32_t mf = *minfar;
    if (mf == 0xffffffffu) return;
    const uint32_t t = mf > 0xffffffffu - delta ? 0xffffffffu : mf + delta;
    if (blockIdx.x == 0 && threadIdx.x == 0) *thresh = t;
    uint32_t n0 = 0, n1 = 0;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        const uint32_t word = a.far_bits[w];
        if (!word) continue;
        uint32_t x = word, promo = 0;
        while (x) {
            const int b = __ffs(x) - 1;
            x &= x - 1;
            if (a.val[32 * w + b] < t) promo |= 1u << b;
        }
        if (!promo) continue;
        a.far_bits[w] = word & ~promo;
        a.bitmap[w] |= promo;
        const uint32_t v0 = 32 * w;
        const uint32_t smask = v0 + 32 <= a.S ? 0xffffffffu : (v0 >= a.S ? 0 : (1u << (a.S - v0)) - 1u);
        n0 += __popc(promo & smask);
        n1 += __popc(promo & ~smask);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        n0 += __shfl_down_sync(kFull, n0, d);
        n1 += __shfl_down_sync(kFull, n1, d);
    }
    if ((threadIdx.x & 31) == 0) {
        if (n0) atomicAdd(&a.cnt_out[6], n0);
        if (n1) atomicAdd(&a.cnt_out[7], n1);
    }
}

// First frontier of a traversal: one source, or every vertex (CC); sets its
// bits and region counts in the parity-0 block.
__global__ void seed_bits_kernel(RegionArgs a, uint32_t src, uint32_t all, uint32_t nwords) {
    if (!all) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.bitmap[src >> 5] |= 1u << (src & 31);
            if (a.visited) a.visited[src >> 5] |= 1u << (src & 31);
            a.cnt_out[src < a.S ? 6 : 7] = 1;
        }
        return;
    }
    uint32_t n0 = 0, n1 = 0;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        const uint32_t v0 = 32 * w;
        uint32_t m = v0 + 32 <= a.V ? 0xffffffffu : (v0 < a.V ? (1u << (a.V - v0)) - 1u : 0);
        a.bitmap[w] = m;
        uint32_t smask = v0 + 32 <= a.S ? 0xffffffffu : (v0 >= a.S ? 0 : (1u << (a.S - v0)) - 1u);
        n0 += __popc(m & smask);
        n1 += __popc(m & ~smask);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        n0 += __shfl_down_sync(kFull, n0, d);
        n1 += __shfl_down_sync(kFull, n1, d);
    }
    if ((threadIdx.x & 31) == 0) {
        if (n0) atomicAdd(&a.cnt_out[6], n0);
        if (n1) atomicAdd(&a.cnt_out[7], n1);
    }
}

template <int ALG>
__global__ void init_values_kernel(uint32_t *val, uint32_t V, uint32_t src) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
        val[i] = ALG == kCC ? i : (i == src ? 1u : V + 1u);
}

// Reached vertices and the sum of their out-degrees (TEPS numerator).
__device__ __forceinline__ void reached_values(const uint32_t *val, const uint32_t *ptr, uint32_t V,
                                               unsigned long long *out) {
    unsigned long long cnt = 0, edges = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
        if (val[i] < V + 1) {
            cnt++;
            edges += ptr[i + 1] - ptr[i];
        }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        cnt += __shfl_down_sync(kFull, cnt, d);
        edges += __shfl_down_sync(kFull, edges, d);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&out[0], cnt);
        atomicAdd(&out[1], edges);
    }
}

__global__ void reached_kernel(const uint32_t *val, const uint32_t *ptr, uint32_t V, unsigned long long *out) {
    reached_values(val, ptr, V, out);
}

// BFS: reached vertices are the reached-vertex bitmap's bits (no level read).
// A warp takes kReachedWords consecutive 32-vertex words at a time, lane =
// vertex: all of their bitmap words and then all the offsets of their reached
// vertices are loaded before any is summed, so each warp keeps several
// independent loads in flight instead of a chain per word.
constexpr int kReachedWords = 4;

__device__ __forceinline__ void reached_bits(const uint32_t *visited, const uint32_t *ptr, uint32_t V,
                                             uint32_t nwords, unsigned long long *out) {
    unsigned long long cnt = 0, edges = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t w0 = kReachedWords * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); w0 < nwords;
         w0 += kReachedWords * warps) {
        uint32_t bits[kReachedWords], lo[kReachedWords], hi[kReachedWords];
#pragma unroll
        for (int k = 0; k < kReachedWords; k++) bits[k] = w0 + k < nwords ? visited[w0 + k] : 0u;
#pragma unroll
        for (int k = 0; k < kReachedWords; k++) {
            const uint32_t v = 32 * (w0 + k) + lane;
            const bool in = ((bits[k] >> lane) & 1u) && v < V;
            lo[k] = in ? ptr[v] : 0u;
            hi[k] = in ? ptr[v + 1] : 0u;
            cnt += in;
        }
#pragma unroll
        for (int k = 0; k < kReachedWords; k++) edges += hi[k] - lo[k];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        cnt += __shfl_down_sync(kFull, cnt, d);
        edges += __shfl_down_sync(kFull, edges, d);
    }
    if (lane == 0 && (cnt | edges)) {
        atomicAdd(&out[0], cnt);
        atomicAdd(&out[1], edges);
    }
}

__global__ void reached_bits_kernel(const uint32_t *visited, const uint32_t *ptr, uint32_t V, uint32_t nwords,
                                    unsigned long long *out) {
    reached_bits(visited, ptr, V, nwords, out);
}

// ------------------------------------------------------- persistent loop -----
//
// A whole traversal in one cooperative launch: set-up, every iteration
// (expansion or bottom-up step, then the next frontier's lists) and the reached
// counts, with a barrier over the grid between phases. An iteration as separate
// launches was five graph nodes, two of them clears, around a few microseconds
// of work when the frontier is small: BFS on 1,001 vertices, 5 iterations, 111 us
// as a CUDA graph of launches and 48 so; RMAT scale 24, 9 iterations, 706 and 651.
// CTAs per SM (registers 48 / 40 / 32 / 32): connected components of 6 M vertices
// 3.60 / 3.61 / 3.65 / 3.64 ms at 5 / 6 / 7 / 8, SSSP on RMAT scale 23 2.95 /
// 2.94 / 2.98 / 2.98, BFS on scale 24 685 / 651 / 658 / 658 us.
#ifndef ASC_TRAV_BLOCKS
#define ASC_TRAV_BLOCKS 6
#endif
struct LoopArgs {
    FusedArgs x0, x1;       // arguments of an iteration by the parity of its input frontier
    uint32_t *ctl;
    uint32_t *report;       // host: the control block at the end
    uint32_t nwords;
    uint32_t src;           // the first frontier's vertex,
    uint32_t all;           // or every vertex
    uint32_t cap;           // iterations
    uint32_t thresh;        // near-far: the first threshold
    uint32_t delta;         // near-far: step of the next one beyond the smallest far value
    uint32_t count_reached;
    uint32_t *values;       // host: small results too (null: the caller copies them)
    uint32_t first_label;   // connected components: src's label is spread first, the rest follow
    uint32_t first_cap;     // after at most this many iterations
    uint32_t polls;         // of a grid barrier before it gives up
};

constexpr uint32_t kFirstLabelIterations = 32;
// A first label that reaches fewer than this many vertices in its second iteration
// follows a thread (a path, a ring, the corner of a grid): the rest joins then. 131,072
// rings of 8 vertices: 5 iterations from every vertex at once 193 us, after the first
// label's own 5 265, after 2 of them 222.
constexpr uint32_t kFirstLabelLeast = 4;
__host__ __device__ __forceinline__ bool rest_joins(uint32_t it, uint64_t frontier, uint32_t first_cap) {
    return !frontier || it >= first_cap || (it == 2 && frontier < kFirstLabelLeast);
}
// Results of at most this many values come back with the report and are copied
// from there on the host: the copy engine's latency is longer (BFS on 1,001
// vertices: 11 to 14 us of 80).
constexpr uint64_t kReportedValues = 16384;

// Polls of a grid barrier (a read of L2 and a short sleep each) before it gives
// up: tens of seconds, far above any phase.
constexpr uint32_t kBarrierPolls = 1u << 25;
thread_local uint32_t t_barrier_polls = kBarrierPolls;  // tests make a thread's runs give up sooner

// Barrier over the grid: arrivals count up from zero for the whole launch.
// False when the other CTAs did not arrive in time. Where counts is given, the
// CTL_BLOCK words there (16-byte aligned) are read once for the CTA into s_counts:
// with every warp of 912 CTAs reading them for itself, those reads of one line cost
// more than the barrier (an iteration of a BFS that reaches 700 vertices at a time
// on a grid graph of a million: 18 us, 13.5 so).
__device__ __forceinline__ bool grid_barrier(const LoopArgs &l, uint32_t &target, const uint32_t *counts = nullptr,
                                             uint32_t *s_counts = nullptr) {
    uint32_t *ctl = l.ctl;
    __shared__ uint32_t s_ok;
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(ctl + CTL_BARRIER, 1u);
        uint32_t now, polls = 0;
        for (;;) {
            // relaxed: an acquire would empty the L1 that the SM's other CTAs still work in
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(ctl + CTL_BARRIER) : "memory");
            if ((int32_t)(now - target) >= 0 || ++polls > l.polls) break;
            if (polls > 16) __nanosleep(64);
        }
        s_ok = (int32_t)(now - target) >= 0;
        if (!s_ok) atomicExch(ctl + CTL_TIMEOUT, 2u);
        __threadfence();
        if (counts) {
            const uint4 a = __ldcg(reinterpret_cast<const uint4 *>(counts));
            const uint4 b = __ldcg(reinterpret_cast<const uint4 *>(counts) + 1);
            reinterpret_cast<uint4 *>(s_counts)[0] = a;
            reinterpret_cast<uint4 *>(s_counts)[1] = b;
        }
    }
    __syncthreads();
    return s_ok != 0;
}

// Values, bitmaps and the first frontier (parity 0) with its list.
template <int ALG>
__device__ __forceinline__ void loop_setup(const LoopArgs &x) {
    const RegionArgs &a = x.x1.r0;  // writes parity 0
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const uint32_t V = a.V;
    for (uint32_t i = 4 * t; i < V; i += 4 * stride) {
        uint4 q;
        q.x = ALG == kCC ? i : V + 1;
        q.y = ALG == kCC ? i + 1 : V + 1;
        q.z = ALG == kCC ? i + 2 : V + 1;
        q.w = ALG == kCC ? i + 3 : V + 1;
        if (ALG != kCC) {
            if (x.src == i) q.x = 1;
            if (x.src == i + 1) q.y = 1;
            if (x.src == i + 2) q.z = 1;
            if (x.src == i + 3) q.w = 1;
        }
        if (i + 4 <= V) {
            *reinterpret_cast<uint4 *>(a.val + i) = q;
        } else {
            a.val[i] = q.x;
            if (i + 1 < V) a.val[i + 1] = q.y;
            if (i + 2 < V) a.val[i + 2] = q.z;
        }
    }
    for (uint32_t w = t; w < V / 32 + 2; w += stride) {
        uint32_t m = 0;
        if (x.all) m = 32 * w + 32 <= V ? 0xffffffffu : (32 * w < V ? (1u << (V - 32 * w)) - 1u : 0u);
        else if (w == x.src >> 5) m = 1u << (x.src & 31);
        a.bitmap[w] = m;
        x.x0.r0.bitmap[w] = 0;
        if (ALG == kBFS) a.visited[w] = m;
        if (ALG == kSSSP && a.far_bits) a.far_bits[w] = 0;
    }
    if (blockIdx.x == 0 && x.all) {
        if (threadIdx.x == 0) {
            a.cnt_out[6] = a.S;
            a.cnt_out[7] = V - a.S;
        }
    } else if (blockIdx.x == 0) {
        const uint32_t deg = a.ptr[x.src + 1] - a.ptr[x.src], od = x.src >= a.S;
        const uint32_t nseg = deg > a.huge ? (deg + a.seg_len - 1) / a.seg_len : 0;
        for (uint32_t k = threadIdx.x; k < nseg; k += blockDim.x)
            a.seg_out[(od ? a.segcap_static : 0) + k] = ((uint64_t)x.src << 32) | k;
        if (threadIdx.x == 0) {
            a.cnt_out[6 + od] = 1;
            a.cnt_out[2 + od] = nseg;
            a.cnt_out[od] = nseg ? 0 : 1;
            if (!nseg) a.q_out[od ? a.S : 0] = x.src;
        }
    }
}

// Near-far: the far vertices below thresh join the frontier in bits (their
// numbers per region are added to moved[0..1]), the smallest value of those that
// stay goes to *minfar.
__device__ __forceinline__ void promote_far(const RegionArgs &a, uint32_t *bits, uint32_t *moved, uint32_t nwords,
                                            uint32_t thresh, uint32_t *minfar) {
    uint32_t n0 = 0, n1 = 0, least = 0xffffffffu;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        const uint32_t word = a.far_bits[w];
        uint32_t x = word, promo = 0;
        while (x) {
            const int b = __ffs(x) - 1;
            x &= x - 1;
            const uint32_t val = a.val[32 * w + b];
            if (val < thresh) promo |= 1u << b;
            else least = min(least, val);
        }
        if (!promo) continue;
        a.far_bits[w] = word & ~promo;
        bits[w] |= promo;
        const uint32_t v0 = 32 * w;
        const uint32_t smask = v0 + 32 <= a.S ? 0xffffffffu : (v0 >= a.S ? 0 : (1u << (a.S - v0)) - 1u);
        n0 += __popc(promo & smask);
        n1 += __popc(promo & ~smask);
    }
    n0 = __reduce_add_sync(kFull, n0);
    n1 = __reduce_add_sync(kFull, n1);
    least = __reduce_min_sync(kFull, least);
    if ((threadIdx.x & 31) == 0) {
        if (n0) atomicAdd(&moved[0], n0);
        if (n1) atomicAdd(&moved[1], n1);
        if (least != 0xffffffffu) atomicMin(minfar, least);
    }
}

// Connected components, once the first label is spread: every other vertex with
// out-edges that kept its own id joins the frontier in bits (their numbers per
// region are added to moved[0..1]).
__device__ __forceinline__ void seed_unlabelled(const RegionArgs &a, uint32_t *bits, uint32_t src, uint32_t *moved) {
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * kWarps;
    uint32_t n0 = 0, n1 = 0;
    for (uint32_t w = blockIdx.x * kWarps + (threadIdx.x >> 5); 32 * w < a.V; w += warps) {
        const uint32_t v = 32 * w + lane;
        const bool join = v < a.V && v != src && a.val[v] == v && a.ptr[v + 1] != a.ptr[v];
        const uint32_t word = __ballot_sync(kFull, join) | bits[w];
        if (lane == 0 && word) {
            bits[w] = word;
            const uint32_t smask = 32 * w + 32 <= a.S ? 0xffffffffu : (32 * w >= a.S ? 0 : (1u << (a.S - 32 * w)) - 1u);
            n0 += __popc(word & smask);
            n1 += __popc(word & ~smask);
        }
    }
    if (lane == 0 && n0) atomicAdd(&moved[0], n0);
    if (lane == 0 && n1) atomicAdd(&moved[1], n1);
}

__global__ void seed_unlabelled_kernel(RegionArgs a, uint32_t *bits, uint32_t src, uint32_t *moved) {
    seed_unlabelled(a, bits, src, moved);
}

struct LoopState {
    uint32_t target = 0;      // of the grid barrier
    uint32_t it = 0;
    uint32_t thresh = 0;
    uint32_t promotions = 0;
};

enum LoopNext { kLoopGo, kLoopEnd, kLoopStuck };

template <int WORDS>
union LoopSmem {
    ExpandSmem<WORDS> expand;
    BuSmem bottom_up;
};

// One iteration from the frontier that x reads; y's arguments write that
// frontier's lists (the other parity). cin: shared, its counts; the next one's
// when the iteration ends.
template <int ALG, int WORDS>
__device__ __forceinline__ LoopNext loop_iteration(const LoopArgs &l, const FusedArgs &x, const FusedArgs &y,
                                                   LoopState &st, LoopSmem<WORDS> &sm, uint32_t *s_next,
                                                   uint32_t *cin) {
    const RegionArgs &a = x.r0;
    if (ALG == kCC && l.first_label && !st.promotions &&
        rest_joins(st.it, (uint64_t)cin[6] + cin[7], l.first_cap)) {
        // the frontier of the remaining labels, in place of an empty one or beside
        // what the first label still has to reach
        st.promotions = 1;
        if (!grid_barrier(l, st.target)) return kLoopStuck;  // every thread has read the counts
        if (blockIdx.x == 0 && threadIdx.x < CTL_BLOCK) y.r0.cnt_out[threadIdx.x] = 0;
        seed_unlabelled(a, y.r0.bitmap, l.src, l.ctl + CTL_PROMOTED);
        if (!grid_barrier(l, st.target, l.ctl + CTL_PROMOTED, cin)) return kLoopStuck;
        const uint32_t n0 = cin[0], n1 = cin[1];
        build_frontier(y.r0, y.r0.bitmap, l.nwords, n0, n1);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            y.r0.cnt_out[6] = n0;
            y.r0.cnt_out[7] = n1;
        }
        if (!grid_barrier(l, st.target, a.cnt_in, cin)) return kLoopStuck;
    }
    if (!(cin[6] | cin[7])) {
        if (ALG != kSSSP || !a.far_bits) return kLoopEnd;
        // The near frontier is empty: the threshold moves on. Every promotion
        // counts in a slot of its own (of four; the one after next is cleared), and
        // the frontier's counts are set only once every thread has read them as zero.
        uint32_t n0, n1;
        for (;;) {
            const uint32_t k = st.promotions++ & 3, clear = (k + 2) & 3;
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                l.ctl[CTL_MINFAR + clear] = 0xffffffffu;
                l.ctl[CTL_PROMOTED + 2 * clear] = l.ctl[CTL_PROMOTED + 2 * clear + 1] = 0;
            }
            promote_far(a, y.r0.bitmap, l.ctl + CTL_PROMOTED + 2 * k, l.nwords, st.thresh, l.ctl + CTL_MINFAR + k);
            if (!grid_barrier(l, st.target)) return kLoopStuck;
            volatile const uint32_t *moved = l.ctl + CTL_PROMOTED + 2 * k;
            n0 = moved[0];
            n1 = moved[1];
            if (n0 | n1) break;
            const uint32_t least = *(volatile uint32_t *)(l.ctl + CTL_MINFAR + k);
            if (least == 0xffffffffu) return kLoopEnd;
            st.thresh = least > 0xffffffffu - l.delta ? 0xffffffffu : least + l.delta;
        }
        build_frontier(y.r0, y.r0.bitmap, l.nwords, n0, n1);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            y.r0.cnt_out[6] = n0;
            y.r0.cnt_out[7] = n1;
        }
        if (!grid_barrier(l, st.target, a.cnt_in, cin)) return kLoopStuck;
    }
    if (st.it >= l.cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) l.ctl[CTL_TIMEOUT] = 1;
        return kLoopEnd;
    }
    st.it++;
    if (ALG == kBFS && bottom_up_step(a, cin)) bottom_up_words(a, l.nwords, st.it + 1, sm.bottom_up, s_next);
    else expand_regions<ALG, WORDS>(x, cin, st.thresh, sm.expand, s_next);
    if (!grid_barrier(l, st.target, a.cnt_out, cin)) return kLoopStuck;
    build_frontier(a, a.bitmap, l.nwords, cin[6], cin[7]);
    // the input frontier's bitmap and counts are the next output's
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < l.nwords; w += gridDim.x * blockDim.x)
        y.r0.bitmap[w] = 0;
    if (blockIdx.x == 0 && threadIdx.x < CTL_BLOCK) y.r0.cnt_out[threadIdx.x] = 0;
    return grid_barrier(l, st.target, a.cnt_out, cin) ? kLoopGo : kLoopStuck;
}

template <int ALG, int WORDS>
__global__ void __launch_bounds__(kBlock, ASC_TRAV_BLOCKS) traverse_kernel(const __grid_constant__ LoopArgs l) {
    __shared__ LoopSmem<WORDS> sm;
    __shared__ uint32_t s_next[kNextWords];
    __shared__ alignas(16) uint32_t cin[CTL_BLOCK];
    LoopState st;
    st.thresh = l.thresh;
    loop_setup<ALG>(l);
    if (!grid_barrier(l, st.target, l.x0.r0.cnt_in, cin)) return;
    if (l.all) {
        build_frontier(l.x1.r0, l.x1.r0.bitmap, l.nwords, cin[6], cin[7]);
        if (!grid_barrier(l, st.target, l.x0.r0.cnt_in, cin)) return;
    }
    for (;;) {
        LoopNext n = loop_iteration<ALG, WORDS>(l, l.x0, l.x1, st, sm, s_next, cin);
        if (n == kLoopGo) n = loop_iteration<ALG, WORDS>(l, l.x1, l.x0, st, sm, s_next, cin);
        if (n == kLoopStuck) return;
        if (n == kLoopEnd) break;
    }
    unsigned long long *out = (unsigned long long *)(l.ctl + CTL_STATS) + 4;
    if (l.count_reached) {
        if (ALG == kBFS) reached_bits(l.x0.r0.visited, l.x0.r0.ptr, l.x0.r0.V, l.nwords, out);
        else reached_values(l.x0.r0.val, l.x0.r0.ptr, l.x0.r0.V, out);
    }
    if (l.values)
        for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < l.x0.r0.V; v += gridDim.x * blockDim.x)
            l.values[v] = l.x0.r0.val[v];
    if (!grid_barrier(l, st.target)) return;
    if (blockIdx.x == 0 && threadIdx.x < CTL_WORDS)
        l.report[threadIdx.x] = threadIdx.x == CTL_ITERS ? st.it : ((volatile uint32_t *)l.ctl)[threadIdx.x];
}

// ------------------------------------------------------------- PageRank -----
//
// Ranks are FP64 in every mode; the contributions rank/outDeg that the edges
// carry are T (FP64, or FP32 for the precision pattern: 4 bytes per edge
// gather, and half the L2 footprint of the contribution array).
//
// How the sums of contributions accumulate (PrAcc<T>): FP64 contributions add
// in FP64, where the order of the atomics changes a sum by about 1e-16
// relative, far below the stop tolerance. FP32 contributions add in FP32 only
// in a fixed order (a thread's own edges, then a warp's segmented shuffle
// tree), and every partial that meets others through an atomic (across warps,
// tiles, segments or a scatter's edges) adds exactly, as 64-bit fixed point
// with 62 fraction bits. Integer addition is associative, so the atomics'
// order cannot change a sum: every pass recomputes bit-identical sums from
// identical contributions, and the FP64 L1 residual falls to the stop
// tolerance. (FP32 atomics in any order floor it near 1.5e-8 at RMAT scale
// 25, so that such a run always took the pass cap.) A sum is at most the total
// rank (1 in standard mode), so two integer bits are enough; a partial below
// 2^-62 rounds to the grid (an absolute error below 1.1e-19 each).
template <typename T>
struct PrAcc;
template <>
struct PrAcc<double> {
    typedef double type;
    static __device__ __forceinline__ double from(double x) { return x; }
    static __device__ __forceinline__ double value(double a) { return a; }
};
template <>
struct PrAcc<float> {
    typedef unsigned long long type;
    static __device__ __forceinline__ unsigned long long from(float x) { return __float2ull_rn(x * 0x1p62f); }
    static __device__ __forceinline__ double value(unsigned long long a) { return __ull2double_rn(a) * 0x1p-62; }
};

// Arguments of the list-driven passes of reference PageRank.
struct PrArgs {
    RegionArgs r;           // lists, segments, counts (pull over in-edges)
    const uint32_t *outdeg;
    double *rank;
    const double *c_old;
    double *c_new;
    double *sum;            // partial sums of segmented vertices
};

// The reference update of an active vertex from its sum s (prKernel_Opt,
// gpu_kernels.cuh:533-552): true while it stays active.
__device__ __forceinline__ bool pr_ref_row(double *rank, const double *c_old, double *c_new, uint32_t v, uint32_t od,
                                           double s) {
    const double r = rank[v];
    const double t = fma(0.85, s, 0.15);
    const double diff = t > r ? t - r : r - t;
    if (diff > 0.001) {
        rank[v] = t;
        c_new[v] = od ? t / (double)od : 0.0;
        return true;
    }
    c_new[v] = c_old[v];
    return false;
}

__device__ __forceinline__ void block_reduce2_atomic(double a, double b, double *out, double *s_buf) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        a += __shfl_down_sync(kFull, a, d);
        b += __shfl_down_sync(kFull, b, d);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        s_buf[2 * w] = a;
        s_buf[2 * w + 1] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double x = 0, y = 0;
        for (int i = 0; i < kWarps; i++) {
            x += s_buf[2 * i];
            y += s_buf[2 * i + 1];
        }
        if (x != 0) atomicAdd(&out[0], x);
        if (y != 0) atomicAdd(&out[1], y);
    }
    __syncthreads();
}

// Edges per thread per pass of the PageRank pull (all reads issued first).
#ifndef ASC_PR_UNROLL
#define ASC_PR_UNROLL 4
#endif
constexpr int kPrUnroll = ASC_PR_UNROLL;
struct PrSmem {
    uint32_t pref[kBlock + 1];
    uint32_t start[kBlock];
    uint32_t warp[kWarps + 1];
    double sum[kBlock];
    uint32_t work;
};

// A tile of active vertices of a reference pass, which walks the active set
// like a traversal frontier (list, or the bitmap in id order when dense); a
// vertex that stays active sets its bit in the next bitmap.
__device__ void pr_vertices(const PrArgs &p, bool valid, uint32_t u, PrSmem &sm, uint32_t *s_next) {
    const RegionArgs &a = p.r;
    uint32_t deg = 0, start = 0;
    bool huge = false;
    if (valid) {
        start = a.ptr[u];
        deg = a.ptr[u + 1] - start;
        huge = deg > a.huge;
        if (huge) deg = 0;
    }
    uint32_t total;
    uint32_t excl = block_excl_scan(deg, total, sm.warp);
    sm.pref[threadIdx.x] = excl;
    sm.start[threadIdx.x] = start;
    sm.sum[threadIdx.x] = 0;
    if (threadIdx.x == 0) sm.pref[kBlock] = total;
    const uint32_t nact = __syncthreads_count(valid && !huge);
    const int lane = threadIdx.x & 31;
    // kPrUnroll edges per thread per pass (edge k of a pass is edge
    // base + k * kBlock + thread): every source id is loaded, then every
    // contribution gathered, before any is summed, so a thread has kPrUnroll
    // reads in flight instead of one
    for (uint32_t base = 0; base < total; base += kPrUnroll * kBlock) {
        double x[kPrUnroll];
        int owner[kPrUnroll];
        uint32_t srcv[kPrUnroll];
#pragma unroll
        for (int k = 0; k < kPrUnroll; k++) {
            const uint32_t e = base + k * kBlock + threadIdx.x;
            owner[k] = -1 - lane;  // distinct per invalid lane
            srcv[k] = 0xffffffffu;
            if (e < total) {
                int lo = 0, hi = kBlock;
                while (hi - lo > 1) {
                    int mid = (lo + hi) >> 1;
                    if (sm.pref[mid] <= e) lo = mid;
                    else hi = mid;
                }
                owner[k] = lo;
                srcv[k] = edge_word(a.edges, (uint64_t)sm.start[lo] + (e - sm.pref[lo]), a.ebits);
                if (ASC_BAD(srcv[k] >= a.V, 21, srcv[k])) {
                    srcv[k] = 0xffffffffu;
                    owner[k] = -1 - lane;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kPrUnroll; k++) x[k] = srcv[k] != 0xffffffffu ? p.c_old[srcv[k]] : 0.0;
#pragma unroll
        for (int k = 0; k < kPrUnroll; k++) {
            // segmented suffix sum over lanes with the same owner (owners
            // ascend with the lane)
            double xs = x[k];
            const int ow = owner[k];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                double y = __shfl_down_sync(kFull, xs, d);
                int oy = __shfl_down_sync(kFull, ow, d);
                if (lane + d < 32 && oy == ow) xs += y;
            }
            int oprev = __shfl_up_sync(kFull, ow, 1);
            if (ow >= 0 && (lane == 0 || oprev != ow)) atomicAdd(&sm.sum[ow], xs);
        }
    }
    __syncthreads();
    const bool won =
        valid && !huge && pr_ref_row(p.rank, p.c_old, p.c_new, u, p.outdeg[u], sm.sum[threadIdx.x]);
    if (won) atomicOr(&a.bitmap[u >> 5], 1u << (u & 31));
    count_next(a, won, u, s_next);
    const uint32_t e = __reduce_add_sync(kFull, won ? deg : 0u);
    if (lane == 0 && e) atomicAdd(a.stats + (CTL_ACTIVE - CTL_STATS) / 2, (unsigned long long)e);
    if (threadIdx.x == 0) {
        atomicAdd(&a.stats[a.region], (unsigned long long)total);
        atomicAdd(&a.stats[2 + a.region], (unsigned long long)nact);
    }
    __syncthreads();
}

__device__ void pr_segment(const PrArgs &p, uint64_t item, PrSmem &sm) {
    const RegionArgs &a = p.r;
    const uint32_t u = (uint32_t)(item >> 32), k = (uint32_t)item;
    const uint32_t b0 = a.ptr[u], e0 = a.ptr[u + 1];
    const uint64_t b = (uint64_t)b0 + (uint64_t)k * a.seg_len;
    const uint64_t e = min((uint64_t)e0, b + a.seg_len);
    const uint32_t n = (uint32_t)(e - b);
    double x = 0;
    for (uint32_t j0 = threadIdx.x; j0 < n; j0 += kPrUnroll * kBlock) {
        // kPrUnroll loads in flight, added in edge order
        uint32_t sv[kPrUnroll];
#pragma unroll
        for (int k = 0; k < kPrUnroll; k++) {
            const uint32_t j = j0 + k * kBlock;
            sv[k] = j < n ? edge_word(a.edges, b + j, a.ebits) : 0xffffffffu;
            if (sv[k] != 0xffffffffu && ASC_BAD(sv[k] >= a.V, 21, sv[k])) sv[k] = 0xffffffffu;
        }
        double c[kPrUnroll];
#pragma unroll
        for (int k = 0; k < kPrUnroll; k++) c[k] = sv[k] != 0xffffffffu ? p.c_old[sv[k]] : 0.0;
#pragma unroll
        for (int k = 0; k < kPrUnroll; k++)
            if (sv[k] != 0xffffffffu) x += c[k];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x += __shfl_down_sync(kFull, x, d);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sm.sum[w] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0;
        for (int i = 0; i < kWarps; i++) s += sm.sum[i];
        atomicAdd(&p.sum[u], s);
        atomicAdd(&a.stats[a.region], (unsigned long long)n);
        if (k == 0) atomicAdd(&a.stats[2 + a.region], 1ull);
    }
    __syncthreads();
}

__device__ __forceinline__ void pr_list_item(const PrArgs &p, uint32_t w, uint32_t n_in, uint32_t nseg, bool bitmap,
                                             uint32_t per, PrSmem &sm, uint32_t *s_next) {
    const RegionArgs &a = p.r;
    if (w < nseg) {
        pr_segment(p, a.seg_in[w], sm);
    } else if (bitmap) {
        const uint32_t u = (a.dense_begin & ~31u) + (w - nseg) * kBlock + threadIdx.x;
        const bool valid = (region_word(a, u & ~31u) >> (u & 31)) & 1u;
        if (__syncthreads_or(valid)) pr_vertices(p, valid, u, sm, s_next);
    } else {
        const uint32_t i = (w - nseg) * per + threadIdx.x;
        const bool valid = threadIdx.x < per && i < n_in;
        pr_vertices(p, valid, valid ? a.q_in[i] : 0u, sm, s_next);
    }
}

// Both regions of a list-driven pass in one launch, items alternating between
// the on-demand and the static region while both have some (as the traversal's
// fused expansion), so every SM overlaps host-link reads with HBM reads.
// regions: bit 0 static, bit 1 on-demand.
__global__ void __launch_bounds__(kBlock, ASC_PR_MIN_BLOCKS) pr_pull_lists_kernel(PrArgs p0, PrArgs p1,
                                                                                  uint32_t regions) {
    __shared__ PrSmem sm;
    __shared__ uint32_t s_next[2];
    if (threadIdx.x < 2) s_next[threadIdx.x] = 0;
    uint32_t n0, s0, i0, t0, n1, s1, i1, t1;
    bool b0, b1;
    region_items_bits(p0.r, p0.r.cnt_in, n0, s0, i0, b0, t0);
    region_items_bits(p1.r, p1.r.cnt_in, n1, s1, i1, b1, t1);
    if (!(regions & 1u)) i0 = 0;
    if (!(regions & 2u)) i1 = 0;
    const uint32_t m = min(i0, i1), total = i0 + i1;
    uint32_t *work = (regions & 1u) ? p0.r.work : p1.r.work;
    for (;;) {
        if (threadIdx.x == 0) sm.work = atomicAdd(work, 1u);
        __syncthreads();
        const uint32_t w = sm.work;
        __syncthreads();
        if (w >= total) break;
        bool od;
        uint32_t local;
        if (w < 2 * m) {
            od = (w & 1) == 0;
            local = w >> 1;
        } else {
            od = i1 > i0;
            local = m + (w - 2 * m);
        }
        if (od) pr_list_item(p1, local, n1, s1, b1, t1, sm, s_next);
        else pr_list_item(p0, local, n0, s0, b0, t0, sm, s_next);
    }
    flush_next(p0.r, s_next);
}

// Applies the segmented vertices once all their segments are summed (this
// pass's segment items; k == 0 marks the vertex).
__global__ void pr_apply_segmented_kernel(PrArgs p, const uint64_t *items_static, const uint64_t *items_od) {
    const RegionArgs &a = p.r;
    const uint32_t n0 = a.cnt_in[2], n = n0 + a.cnt_in[3];
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t i = base + threadIdx.x;
        bool won = false;
        uint32_t v = 0;
        if (i < n) {
            const uint64_t it = i < n0 ? items_static[i] : items_od[i - n0];
            v = (uint32_t)(it >> 32);
            if ((uint32_t)it == 0) {
                const double s = p.sum[v];
                p.sum[v] = 0;
                won = pr_ref_row(p.rank, p.c_old, p.c_new, v, p.outdeg[v], s);
            }
        }
        // a long-list vertex that stays active joins the next bitmap
        if (won) {
            atomicOr(&a.bitmap[v >> 5], 1u << (v & 31));
            atomicAdd(a.stats + (CTL_ACTIVE - CTL_STATS) / 2, (unsigned long long)(a.ptr[v + 1] - a.ptr[v]));
        }
        const unsigned m0 = __ballot_sync(kFull, won && v < a.S), m1 = __ballot_sync(kFull, won && v >= a.S);
        if ((threadIdx.x & 31) == 0) {
            if (m0) atomicAdd(&a.cnt_out[6], (uint32_t)__popc(m0));
            if (m1) atomicAdd(&a.cnt_out[7], (uint32_t)__popc(m1));
        }
    }
}

// ------------------------------------------- edge-balanced PageRank passes --
//
// A standard pass runs over the merge items (kItem positions each). Tiles of 256
// vertices held from none to 131,000 edges (lists of up to 512 each), every edge
// searched its owner in shared memory, and a segmented 5-step shuffle sum ran
// per edge: 197 instructions per edge (ncu, FP64 pull, 25.5 M edges), with 5 FP64
// adds per edge on a pipe that takes 16 cycles per warp instruction.
//
// Here every row that ends in the item marks its last edge, a thread takes
// kVt consecutive edges and closes a sum at each mark, and one segmented warp
// scan joins the sums of rows that cross threads: one add per edge and no
// search. Bound by the host link (30% resident: 2.29 of the 2.5 ms a pass takes
// on RMAT scale 24, FP32; 172 of 215 us on 25.5 M edges, FP64).
// Standard PageRank to 1e-9 before / after: FP32, RMAT scale 24, 101.0 / 73.5 ms
// (its passes 3.26 / 2.53 ms); FP64, 1.5 M vertices of degree 17, 11.5 / 5.06 ms.
// CTAs of 256 threads, 6 per SM: 73.5 and 5.06 ms; 128 threads, 12 per SM: 75.2
// and 5.06 (8 per SM: 77.7, 5.10); 64 threads, 24 per SM: 104.3, 5.25. Shared
// memory of more CTAs takes the L1 that holds the gathers in flight: 14 CTAs of
// 128 threads measured 121.7 and 8.1 ms.
#ifndef ASC_PR_ITEM_BLOCKS
#define ASC_PR_ITEM_BLOCKS 6
#endif
// A reference-mode pass runs over all items while the active vertices hold more
// than 1 / kPrDenseDiv of the in-edges, else over their lists. 35 passes on RMAT
// scale 20 (85% of the edges active on average), 30% resident: lists alone 11.15
// ms; items above 1/2, 1/4, 1/8, 1/32 and always: 5.25, 5.38, 5.38, 5.47, 5.55.
#ifndef ASC_PR_DENSE_DIV
#define ASC_PR_DENSE_DIV 2
#endif
constexpr uint64_t kPrDenseDiv = ASC_PR_DENSE_DIV;
// Scatter passes: slots for hot destinations and CTAs per SM (see pr_hot_slot).
#ifndef ASC_PR_HOT
#define ASC_PR_HOT 1024
#endif
#ifndef ASC_PR_SCATTER_BLOCKS
#define ASC_PR_SCATTER_BLOCKS 4
#endif
constexpr uint32_t kPrHot = ASC_PR_HOT;

// A range of items and where their edges are read.
struct PrSlice {
    const uint32_t *edges;   // indexed by global edge offset
    uint64_t edge_words;     // words that may be read there
    uint32_t begin, n;       // items [begin, begin + n)
};

template <typename T>
struct PrItemArgs {
    typedef typename PrAcc<T>::type Acc;
    const uint2 *items;
    PrSlice sl[2];           // static, on-demand
    const uint32_t *ptr;
    const uint32_t *outdeg;
    double *rank;
    const T *c_old;
    T *c_new;
    Acc *sum;                // sums of the rows cut by item boundaries (zero between passes)
    double damping;
    const double *dangling_prev;   // dangling mass of the previous pass
    double *acc;             // [0] residual, [1] dangling of this pass
    uint32_t *work;
    uint32_t V, ebits;
    uint32_t wbits;          // scatter: weight bits below the destination in an edge word
    const unsigned long long *hot;  // scatter: hot destinations by slot
    const uint32_t *active_prev;    // scatter, reference mode: vertices the previous pass left active
    // reference mode: active vertices of this pass and the next one, their counts
    // per region (cnt_out[6..7]) and the next one's in-edges
    const uint32_t *bitmap_in;
    uint32_t *bitmap, *cnt_in, *cnt_out;
    unsigned long long *active_edges;
    uint32_t S;
    // how a pass ends (see pr_pass_over)
    const double *res_prev;  // residual of the previous pass (null: first pass)
    double tolerance;
    double *acc_next;        // cleared for the next pass
    uint32_t *ticket;
    unsigned long long *report;  // host: residual, or active vertices (2) and in-edges
};

template <typename T>
struct PrItemSmem {
    // the item's edge words, then its row sums: at most ne words and 2 (nr + 1)
    // words with nr + ne <= kItem, plus alignment and one word read past the end
    alignas(16) uint32_t pool[2 * kItem + 16];
    uint16_t row_at[kItem];       // of an edge that ends a row: the row, from the item's first
    uint32_t marks[2][kItem / 32];  // one bit per edge: it ends a row (this item's, the next one's)
    double red[2 * kWarps];
    double base;
    uint32_t work[2];
};

// Marks the rows that end in an item (r0 .. r0 + nr - 1, edges from e0) at
// their last edges; rows without edges have none. Every thread calls it.
template <typename T>
__device__ __forceinline__ void pr_mark_rows(const uint32_t *ptr, uint32_t r0, uint32_t e0, uint32_t nr,
                                             PrItemSmem<T> &sm, uint32_t *marks) {
    for (uint32_t j = threadIdx.x; j < nr; j += kBlock) {
        const uint32_t lo = max(ptr[r0 + j], e0), hi = ptr[r0 + j + 1];
        if (hi > lo) {
            const uint32_t x = hi - 1 - e0;
            sm.row_at[x] = (uint16_t)j;
            atomicOr(&marks[x >> 5], 1u << (x & 31));
        }
    }
}

// The row of the first mark at or after edge xe (a multiple of 32), or nr (the
// row that goes on past the item) when there is none. The whole warp calls it.
__device__ __forceinline__ uint32_t pr_next_row(const uint32_t *marks, const uint16_t *row_at, uint32_t xe,
                                                uint32_t nr) {
    const int lane = threadIdx.x & 31;
    for (uint32_t m0 = xe >> 5; m0 < kItem / 32; m0 += 32) {
        const uint32_t word = m0 + lane < kItem / 32 ? marks[m0 + lane] : 0u;
        const unsigned any = __ballot_sync(kFull, word != 0);
        if (any) {
            const int q = __ffs((int)any) - 1;
            const uint32_t bits = __shfl_sync(kFull, word, q);
            return row_at[32 * (m0 + q) + __ffs((int)bits) - 1];
        }
    }
    return nr;
}

// Item w of a launch over both slices: the on-demand and the static slice
// alternate while both have items, so every SM overlaps host-link reads with
// HBM reads.
__device__ __forceinline__ uint32_t pr_slice_item(const PrSlice *sl, uint32_t w, bool &od) {
    const uint32_t i0 = sl[0].n, i1 = sl[1].n, m = min(i0, i1);
    uint32_t local;
    if (w < 2 * m) {
        od = (w & 1) == 0;
        local = w >> 1;
    } else {
        od = i1 > i0;
        local = m + (w - 2 * m);
    }
    return sl[od].begin + local;
}

// The standard update of one vertex from its sum, with the pass's constant part
// (1 - d) / V + d * dangling / V given.
template <typename T>
__device__ __forceinline__ void pr_std_row(double *rank, T *c_new, uint32_t v, uint32_t od, double s, double damping,
                                           double base, double &res, double &dang) {
    const double r = rank[v];
    const double rn = base + damping * s;
    res += fabs(rn - r);
    rank[v] = rn;
    T c = (T)0;
    if (od) c = (T)(rn / (double)od);
    else dang += rn;
    c_new[v] = c;
}

// The host reads how a pass ended one pass late, so that the next one is
// already in flight: a pass that follows the last one changes nothing.
template <bool REF, typename T>
__device__ __forceinline__ bool pr_pass_over(const PrItemArgs<T> &p) {
    if (REF) return !(p.cnt_in[6] | p.cnt_in[7]);
    return p.res_prev && *p.res_prev < p.tolerance;
}

// Run by every block of the kernel that ends a pass: the last one reports to the
// host and clears what the next pass counts in.
template <bool REF, typename T>
__device__ __forceinline__ void pr_end_pass(const PrItemArgs<T> &p) {
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(p.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last || threadIdx.x) return;
    __threadfence();
    volatile unsigned long long *r = p.report;
    if (REF) {
        volatile uint32_t *c = p.cnt_out;
        r[0] = ((unsigned long long)c[7] << 32) | c[6];
        r[1] = *(volatile unsigned long long *)p.active_edges;
        *p.active_edges = 0;
    } else {
        r[0] = *(volatile unsigned long long *)p.acc;
        p.acc_next[0] = p.acc_next[1] = 0;
    }
    for (int i = 0; i < CTL_BLOCK; i++) p.cnt_in[i] = 0;  // the next pass's output counts and cursor
    *p.ticket = 0;
}

// What a thread of an item pass counts over the rows it applies.
struct PrCounts {
    double res = 0, dang = 0;         // standard mode
    uint32_t n0 = 0, n1 = 0;          // reference mode: rows still active, per region,
    unsigned long long edges = 0;     // and their in-edges
};

// Applies row v with sum s. Reference mode (prKernel_Opt, gpu_kernels.cuh:533-552)
// leaves inactive vertices alone: both contribution arrays hold their last value.
template <typename T, bool REF>
__device__ __forceinline__ void pr_item_row(const PrItemArgs<T> &p, uint32_t v, double s, double base, PrCounts &n) {
    if (!REF) {
        pr_std_row<T>(p.rank, p.c_new, v, p.outdeg[v], s, p.damping, base, n.res, n.dang);
        return;
    }
    const uint32_t bit = 1u << (v & 31);
    if (!(p.bitmap_in[v >> 5] & bit)) return;
    if (pr_ref_row((double *)p.rank, (const double *)p.c_old, (double *)p.c_new, v, p.outdeg[v], s)) {
        atomicOr(&p.bitmap[v >> 5], bit);
        if (v < p.S) n.n0++;
        else n.n1++;
        n.edges += p.ptr[v + 1] - p.ptr[v];
    }
}

// Adds a block's counts to the pass's (whole warps call it).
template <bool REF, typename T>
__device__ __forceinline__ void pr_flush_counts(const PrItemArgs<T> &p, PrCounts n, double *s_buf) {
    if (!REF) {
        block_reduce2_atomic(n.res, n.dang, p.acc, s_buf);
        return;
    }
    n.n0 = __reduce_add_sync(kFull, n.n0);
    n.n1 = __reduce_add_sync(kFull, n.n1);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) n.edges += __shfl_down_sync(kFull, n.edges, d);
    if ((threadIdx.x & 31) == 0) {
        if (n.n0) atomicAdd(&p.cnt_out[6], n.n0);
        if (n.n1) atomicAdd(&p.cnt_out[7], n.n1);
        if (n.edges) atomicAdd(p.active_edges, n.edges);
    }
}

template <typename T, bool REF>
__global__ void __launch_bounds__(kBlock, ASC_PR_ITEM_BLOCKS) pr_pull_items_kernel(PrItemArgs<T> p) {
    typedef typename PrAcc<T>::type Acc;
    if (pr_pass_over<REF>(p)) return;
    __shared__ PrItemSmem<T> sm;
    const int lane = threadIdx.x & 31;
    const uint32_t total = p.sl[0].n + p.sl[1].n;
    const uint32_t eb = p.ebits, mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
    if (threadIdx.x < kItem / 32) sm.marks[0][threadIdx.x] = sm.marks[1][threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        sm.work[0] = atomicAdd(p.work, 1u);
        if (!REF) sm.base = (1.0 - p.damping) / (double)p.V + p.damping * (*p.dangling_prev) / (double)p.V;
    }
    __syncthreads();
    PrCounts n;
    for (int buf = 0;; buf ^= 1) {
        const uint32_t w = sm.work[buf];
        if (w >= total) break;
        bool od;
        const uint32_t it = pr_slice_item(p.sl, w, od);
        const uint2 a = p.items[it], b = p.items[it + 1];
        const uint32_t r0 = a.x, e0 = a.y, nr = b.x - a.x, ne = b.y - a.y;
        uint32_t nq;
        const uint32_t bit0 = stage_words(p.sl[od].edges, p.sl[od].edge_words, e0, ne, eb, sm.pool, nq);
        Acc *sums = reinterpret_cast<Acc *>(sm.pool + 4 * nq + (nq ? 4 : 0));
        for (uint32_t j = threadIdx.x; j <= nr; j += kBlock) sums[j] = (Acc)0;
        uint32_t *marks = sm.marks[buf];
        pr_mark_rows<T>(p.ptr, r0, e0, nr, sm, marks);
        if (threadIdx.x == 0) sm.work[buf ^ 1] = atomicAdd(p.work, 1u);
        __syncthreads();
        if (threadIdx.x < kItem / 32) sm.marks[buf ^ 1][threadIdx.x] = 0;
        const uint32_t x0 = threadIdx.x * kVt, xw = x0 - lane * kVt;  // first edge of the thread, the warp
        if (xw < ne) {
            T c[kVt];
#pragma unroll
            for (int k = 0; k < kVt; k++) {
                c[k] = (T)0;
                if (x0 + k < ne) {
                    const uint32_t v = staged_word(sm.pool, bit0 + (x0 + k) * eb, mask);
                    if (!ASC_BAD(v >= p.V, 21, v)) c[k] = __ldg(p.c_old + v);
                }
            }
            const uint32_t ends = (marks[x0 >> 5] >> (x0 & 31)) & ((1u << kVt) - 1u);
            // a thread's first sum may go on from earlier threads; later ones are its own
            T part = (T)0, head = (T)0;
#pragma unroll
            for (int k = 0; k < kVt; k++) {
                part += c[k];
                if ((ends >> k) & 1u) {
                    if (ends & ((1u << k) - 1u)) sums[sm.row_at[x0 + k]] = PrAcc<T>::from(part);
                    else head = part;
                    part = (T)0;
                }
            }
            // open sums, scanned over the lanes: a lane with an end starts a new one
            Acc tail = PrAcc<T>::from(part);
            const unsigned ended = __ballot_sync(kFull, ends != 0);
            // lanes since (and with) the last one that starts a sum
            const uint32_t below = ended & (0xffffffffu >> (31 - lane));
            const int run = below ? lane - (31 - __clz((int)below)) : lane + 1;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                if (!__any_sync(kFull, run >= d)) break;
                const Acc y = __shfl_up_sync(kFull, tail, d);
                if (run >= d && lane >= d) tail += y;
            }
            Acc before = __shfl_up_sync(kFull, tail, 1);
            if (lane == 0) before = (Acc)0;
            if (ends) {
                const Acc h = PrAcc<T>::from(head) + before;
                const uint32_t row = sm.row_at[x0 + __ffs((int)ends) - 1];
                // the warp's first row may have begun in another warp
                if (ended & ((1u << lane) - 1u)) sums[row] = h;
                else atomicAdd(&sums[row], h);
            }
            // the warp's last open sum goes to the row that ends after it: the
            // next mark, or the row that goes on past the item
            const uint32_t xe = xw + 32 * kVt;
            if (xe < ne || !((marks[(ne - 1) >> 5] >> ((ne - 1) & 31)) & 1u)) {
                const uint32_t row = pr_next_row(marks, sm.row_at, xe, nr);
                if (lane == 31) atomicAdd(&sums[row], tail);
            }
        }
        __syncthreads();
        // rows that end here are final, but for a first one that began in an
        // earlier item; that one and the row that goes on past the item add to
        // the global sums (pr_cut_rows_kernel applies them)
        const bool cut = p.ptr[r0] < e0;
        const bool goes_on = ne && !((marks[(ne - 1) >> 5] >> ((ne - 1) & 31)) & 1u);
        for (uint32_t j = threadIdx.x; j <= nr; j += kBlock) {
            if (j == nr ? goes_on : (j == 0 && cut)) {
                atomicAdd(&p.sum[r0 + j], sums[j]);
            } else if (j < nr) {
                pr_item_row<T, REF>(p, r0 + j, PrAcc<T>::value(sums[j]), sm.base, n);
            }
        }
        __syncthreads();
    }
    pr_flush_counts<REF>(p, n, sm.red);
}

// Applies the rows that were cut by an item boundary: the row at the start of
// item i, when it began earlier and ends in item i. Ends the pass. Blocks of
// kBlock.
template <typename T, bool REF>
__global__ void pr_cut_rows_kernel(PrItemArgs<T> p, uint32_t n_items) {
    if (pr_pass_over<REF>(p)) return;
    __shared__ double red[2 * kWarps];
    __shared__ double s_base;
    if (!REF && threadIdx.x == 0)
        s_base = (1.0 - p.damping) / (double)p.V + p.damping * (*p.dangling_prev) / (double)p.V;
    __syncthreads();
    PrCounts n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_items; i += gridDim.x * blockDim.x) {
        const uint2 a = p.items[i];
        const uint32_t r_end = p.items[i + 1].x;
        if (r_end > a.x && p.ptr[a.x] < a.y) {
            const double s = PrAcc<T>::value(p.sum[a.x]);
            p.sum[a.x] = 0;
            pr_item_row<T, REF>(p, a.x, s, s_base, n);
        }
    }
    pr_flush_counts<REF>(p, n, red);
    pr_end_pass<REF>(p);
}

// Ends a list-driven reference pass.
template <typename T>
__global__ void pr_end_pass_kernel(PrItemArgs<T> p) {
    pr_end_pass<true>(p);
}

template <typename T>
__global__ void pr_init_kernel(double *rank, T *c0, T *c1, typename PrAcc<T>::type *sum, const uint32_t *outdeg,
                               uint32_t V, double *dang) {
    // dang points at a (residual, dangling) pair; the start vector adds to dangling
    __shared__ double red[2 * kWarps];
    double d = 0;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < V; base += stride) {
        const uint32_t i = base + threadIdx.x;
        if (i < V) {
            const double r = 1.0 / (double)V;
            const uint32_t od = outdeg[i];
            rank[i] = r;
            const T c = od ? (T)(r / (double)od) : (T)0;
            c0[i] = c;
            c1[i] = c;
            sum[i] = 0;
            if (od == 0) d += r;
        }
    }
    block_reduce2_atomic(0.0, d, dang, red);
}

// FP32 results: the FP64 ranks rounded to float (into the caller's device
// buffer, or a staging buffer that is then copied out).
__global__ void pr_rank_to_float_kernel(const double *rank, float *out, uint32_t V) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
        out[i] = (float)rank[i];
}

// --------------------------------------------------------------- host -------

// A graph's tiles are even when none of kBlock vertices holds more than kEvenTiles
// times the mean edges (uniform random graphs, grids, rings: at most 1.2 times; RMAT
// scale 10: 2.3 times, 16: 29, 22: 350).
constexpr uint64_t kEvenTiles = 2;

// Sizes and allocates the frontier machinery of one run for graph g, with
// the graph's tuning or (graph_tuning false) the default thresholds.
asc_status alloc_workspace(asc_graph *g, Workspace *ws, bool graph_tuning = true) {
    ws->V = g->V;
    if (g->has_tuning && graph_tuning) ws->tune = g->tuning;
    ASC_CUDA(cudaDeviceGetAttribute(&ws->num_sms, cudaDevAttrMultiProcessorCount, g->device));
    {
        // persistent grids fill the GPU: as many CTAs per SM as stay resident
        int per_sm = 0;
        ASC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, expand_fused_kernel<kSSSP, 2>, kBlock, 0));
        const uint32_t resident = (uint32_t)std::max(1, per_sm);
        if (!g->has_tuning || !ws->tune.ctas_per_sm || ws->tune.ctas_per_sm > resident) ws->tune.ctas_per_sm = resident;
    }
    const uint64_t V = g->V;
    const uint32_t S = g->static_vertices;
    const Tuning &t = ws->tune;
    std::lock_guard<std::mutex> plan_lk(g->long_lists_mu);
    auto &cache = g->long_lists;
    auto hit = std::find_if(cache.begin(), cache.end(), [&](const asc_graph::LongLists &c) {
        return c.huge_degree == t.huge_degree && c.segment_edges == t.segment_edges;
    });
    if (hit == cache.end()) {
        constexpr size_t kKeep = 4;
        if (cache.size() >= kKeep) cache.erase(cache.begin());
        cache.emplace_back();
        hit = cache.end() - 1;
        asc_graph::LongLists &ll = *hit;
        ll.bits.assign(V / 32 + 2, 0);
        // on host threads, 2^20 vertices each or more (whole bitmap words)
        const uint32_t *ptr = g->h_ptr;
        const uint32_t huge = t.huge_degree, seg = t.segment_edges;
        const uint64_t words = (V + 31) / 32;
        const uint64_t nt = std::max<uint64_t>(
            1, std::min<uint64_t>(std::max(1u, std::thread::hardware_concurrency()), words >> 15));
        std::vector<uint64_t> sums(3 * nt, 0);
        auto scan = [&](uint64_t k) {
            uint64_t n0 = 0, n1 = 0;
            uint32_t tile = 0;
            for (uint64_t w = words * k / nt; w < words * (k + 1) / nt; w++) {
                uint32_t bits = 0;
                if (w % (kBlock / 32) == 0) tile = std::max(tile, ptr[std::min(V, 32 * w + kBlock)] - ptr[32 * w]);
                for (uint64_t v = 32 * w; v < std::min(V, 32 * w + 32); v++) {
                    const uint32_t d = ptr[v + 1] - ptr[v];
                    if (d <= huge) continue;
                    bits |= 1u << (v & 31);
                    (v < S ? n0 : n1) += ((uint64_t)d + seg - 1) / seg;
                }
                ll.bits[w] = bits;
            }
            sums[3 * k] = n0;
            sums[3 * k + 1] = n1;
            sums[3 * k + 2] = tile;
        };
        std::vector<std::thread> threads;
        for (uint64_t k = 1; k < nt; k++) {
            try {
                threads.emplace_back(scan, k);
            } catch (...) {  // no thread to be had
                scan(k);
            }
        }
        scan(0);
        for (auto &th : threads) th.join();
        uint64_t most = 0;  // edges of the fullest tile
        for (uint64_t k = 0; k < nt; k++) {
            ll.seg_static += sums[3 * k];
            ll.seg_ondemand += sums[3 * k + 1];
            most = std::max(most, sums[3 * k + 2]);
        }
        ll.even = most * V <= kEvenTiles * g->E * std::min<uint64_t>(kBlock, V);
        ll.huge_degree = t.huge_degree;
        ll.segment_edges = t.segment_edges;
    }
    const asc_graph::LongLists &ll = *hit;
    const std::vector<uint32_t> &hbits = ll.bits;
    const uint64_t cs = ll.seg_static, co = ll.seg_ondemand;
    ws->segcap_static = cs;
    ws->segcap_ondemand = co;
    ws->item_div = ll.even && g->E >= 8 * V ? 4 : ll.even && g->E >= 3 * V ? 16 : 0xffffffffu;
    uint64_t bytes = 0;
    auto dalloc = [&](void **p, size_t n) -> asc_status {
        n = n ? n : 16;
        ASC_CUDA(cudaMalloc(p, n));
        bytes += n;
        return ASC_OK;
    };
    ASC_TRY(dalloc((void **)&ws->val, 4 * V));
    for (int i = 0; i < 2; i++) ASC_TRY(dalloc((void **)&ws->bitmap[i], 4 * (V / 32 + 2)));
    ASC_TRY(dalloc((void **)&ws->visited, 4 * (V / 32 + 2)));
    ASC_TRY(dalloc((void **)&ws->huge_bits, 4 * (V / 32 + 2)));
    ASC_TRY(dalloc((void **)&ws->far_bits, 4 * (V / 32 + 2)));
    ASC_CUDA(cudaMemcpy(ws->huge_bits, hbits.data(), 4 * (V / 32 + 2), cudaMemcpyHostToDevice));
    for (int i = 0; i < 2; i++) {
        ASC_TRY(dalloc((void **)&ws->queue[i], 4 * V));
        ASC_TRY(dalloc((void **)&ws->segs[i], 8 * (cs + co)));
    }
    ASC_TRY(dalloc((void **)&ws->ctl, 4 * CTL_WORDS));
    ASC_CUDA(cudaHostAlloc((void **)&ws->h_ctl, 4 * (CTL_WORDS + std::min<uint64_t>(V, kReportedValues)),
                           cudaHostAllocDefault));
    for (auto &e : ws->ev) ASC_CUDA(cudaEventCreate(&e));
    ws->device_bytes = bytes;
    return ASC_OK;
}

asc_status ensure_workspace(asc_graph *g) {
    if (g->ws) return ASC_OK;
    g->ws = new Workspace();
    return alloc_workspace(g, g->ws);
}

// PageRank state for contributions of elem bytes: FP64 ranks, two
// contribution arrays (this pass's and the next's), 8-byte sums.
uint64_t pr_buffer_bytes(uint64_t V, size_t elem) { return (16 + 2 * (uint64_t)elem) * V; }

asc_status ensure_pr_buffers(asc_graph *g, size_t elem) {
    Workspace *ws = g->ws;
    if (ws->pr_rank && ws->pr_elem == elem) return ASC_OK;
    for (void *p : {ws->pr_rank, ws->pr_contrib[0], ws->pr_contrib[1], ws->pr_sum})
        if (p) cudaFree(p);
    if (ws->pr_rank && ws->pr_elem) ws->device_bytes -= pr_buffer_bytes(g->V, ws->pr_elem);
    ws->pr_rank = ws->pr_contrib[0] = ws->pr_contrib[1] = ws->pr_sum = nullptr;
    ws->pr_elem = 0;
    ASC_CUDA(cudaMalloc(&ws->pr_rank, 8 * g->V));
    ASC_CUDA(cudaMalloc(&ws->pr_contrib[0], elem * g->V));
    ASC_CUDA(cudaMalloc(&ws->pr_contrib[1], elem * g->V));
    ASC_CUDA(cudaMalloc(&ws->pr_sum, 8 * g->V));
    ws->pr_elem = elem;
    ws->device_bytes += pr_buffer_bytes(g->V, elem);
    return ASC_OK;
}

// A graph's merge items, made once per workspace.
uint64_t items_bytes(uint64_t V, uint64_t E) { return sizeof(uint2) * ((V + E + kItem - 1) / kItem + 2); }

asc_status ensure_items(asc_graph *g, Workspace *ws, cudaStream_t s) {
    if (ws->items) return ASC_OK;
    const uint32_t V = (uint32_t)g->V, S = g->static_vertices;
    // shorter items where a staging buffer is smaller than one (its words, and
    // up to 3 on either side to start and end on 16 bytes)
    const uint64_t bits = g->edge_words == 2 ? 64 : g->ebits;
    uint64_t L = kItem;
    while (g->stage_words && L > 32 && (L * bits + 31) / 32 + 8 > g->stage_words) L /= 2;
    const uint64_t n0 = (S + (uint64_t)g->h_ptr[S] + L - 1) / L, n1 = (V - S + g->E - g->h_ptr[S] + L - 1) / L;
    ASC_CUDA(cudaMalloc((void **)&ws->items, sizeof(uint2) * (n0 + n1 + 1)));
    ws->device_bytes += sizeof(uint2) * (n0 + n1 + 1);
    ws->n_items_static = (uint32_t)n0;
    ws->n_items = (uint32_t)(n0 + n1);
    const uint64_t blocks = std::min<uint64_t>((n0 + n1) / kBlock + 1, (uint64_t)ws->num_sms * 8);
    merge_plan_kernel<<<(uint32_t)blocks, kBlock, 0, s>>>(g->d_ptr, S, V, (uint32_t)L, ws->n_items_static, ws->n_items,
                                                          ws->items);
    ASC_CUDA(cudaGetLastError());
    return ASC_OK;
}

asc_status ensure_items(asc_graph *g) { return ensure_items(g, g->ws, g->stream); }

// How PageRank passes report to the host: pass k writes two words of page-locked
// memory (kPassSlots slots) and an event says when. At most two passes are in
// flight; one at a time where the caller watches iterations.
constexpr int kPassSlots = 4;
unsigned long long *pass_slot(Workspace *ws, int k) {
    return (unsigned long long *)ws->h_ctl + 2 * (k % kPassSlots);
}
asc_status ensure_pass_events(Workspace *ws) {
    for (auto &e : ws->pass_ev)
        if (!e) ASC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return ASC_OK;
}
// The waits of pass k's end and the standard-mode fields of its arguments: the
// residual and dangling-mass pairs of three consecutive passes.
template <typename T>
void set_pass(Workspace *ws, const asc_params &p, int k, PrItemArgs<T> &a) {
    double *acc = (double *)(ws->ctl + CTL_ACC);
    a.acc = acc + 2 * (k % 3);
    a.acc_next = acc + 2 * ((k + 1) % 3);
    const double *prev = acc + 2 * ((k + 2) % 3);
    a.dangling_prev = prev + 1;
    a.res_prev = k ? prev : nullptr;
    a.tolerance = p.tolerance;
    a.damping = p.damping;
    a.ticket = ws->ctl + CTL_TICKET;
    a.report = pass_slot(ws, k);
}

// A region's items and edges.
PrSlice pr_slice(const asc_graph *g, int region) {
    const Workspace *ws = g->ws;
    PrSlice x;
    x.edges = region == 0 ? g->d_static : g->d_host_edges;
    x.edge_words = edge_store_words(g, region == 0 ? g->static_edges : g->E);
    x.begin = region == 0 ? 0 : ws->n_items_static;
    x.n = region == 0 ? ws->n_items_static : ws->n_items - ws->n_items_static;
    return x;
}

// Edges (static, on-demand) and vertices (likewise) of passes that read every edge.
void pr_pass_counts(const asc_graph *g, uint64_t passes, unsigned long long n[4]) {
    const uint64_t se = g->h_ptr[g->static_vertices];
    n[0] = passes * se;
    n[1] = passes * (g->E - se);
    n[2] = passes * g->static_vertices;
    n[3] = passes * (g->V - g->static_vertices);
}

RegionArgs base_args(asc_graph *g, Workspace *ws, int parity_in) {
    RegionArgs a;
    memset(&a, 0, sizeof(a));
    a.ptr = g->d_ptr;
    a.val = ws->val;
    a.bitmap = ws->bitmap[1 - parity_in];
    a.bitmap_in = ws->bitmap[parity_in];
    a.visited = ws->visited;
    a.huge_bits = ws->huge_bits;
    a.dense_div = ws->tune.dense_div;
    a.wbits = g->wbits;
    a.ebits = g->edge_words == 1 ? g->ebits : 32;
    a.frag = ws->frag_active;
    if (ws->bu_active && ws->in_ptr) {
        a.in_ptr = ws->in_ptr;
        a.in_edges = ws->in_edges ? ws->in_edges : g->d_host_in_edges;
        a.in_resident = ws->in_edges != nullptr;
        a.in_heads = g->in_heads_ready ? g->d_in_heads : nullptr;
        a.in_none = ws->in_none;
        a.in_ebits = g->in_ebits;
        a.bu_div = ws->tune.bu_div;
    }
    a.S = g->static_vertices;
    a.V = (uint32_t)g->V;
    a.huge = ws->tune.huge_degree;
    a.seg_len = ws->tune.segment_edges;
    a.segcap_static = (uint32_t)ws->segcap_static;
    a.segcap_ondemand = (uint32_t)ws->segcap_ondemand;
    a.stats = (unsigned long long *)(ws->ctl + CTL_STATS);
    const int po = 1 - parity_in;
    a.cnt_in = ws->ctl + CTL_BLOCK * parity_in;
    a.cnt_out = ws->ctl + CTL_BLOCK * po;
    a.q_out = ws->queue[po];
    a.seg_out = ws->segs[po];
    return a;
}

RegionArgs base_args(asc_graph *g, int parity_in) { return base_args(g, g->ws, parity_in); }

RegionArgs region_args(asc_graph *g, Workspace *ws, int parity_in, int region, bool dense) {
    RegionArgs a = base_args(g, ws, parity_in);
    a.region = region;
    a.edges = region == 0 ? g->d_static : g->d_host_edges;
    a.dense_begin = region == 0 ? 0 : g->static_vertices;
    a.dense_end = region == 0 ? g->static_vertices : (uint32_t)g->V;
    if (dense) {
        a.q_in = nullptr;
    } else {
        a.q_in = ws->queue[parity_in] + (region == 0 ? 0 : g->static_vertices);
    }
    a.seg_in = ws->segs[parity_in] + (region == 0 ? 0 : ws->segcap_static);
    a.work = a.cnt_out + 4 + region;
    a.edge_words = region == 0 ? edge_store_words(g, g->static_edges) : edge_store_words(g, g->E);
    return a;
}

RegionArgs region_args(asc_graph *g, int parity_in, int region, bool dense) {
    return region_args(g, g->ws, parity_in, region, dense);
}

// SSSP near-far on: the expansion parks distances at or above the threshold in
// the far set.
bool near_far(asc_graph *g, asc_algo algo) { return algo == ASC_SSSP && g->ws->tune.delta != 0; }

void attach_items(const Workspace *ws, RegionArgs &a) {
    a.items = ws->items;
    a.item_div = ws->item_div;
    a.item_begin = a.region == 0 ? 0 : ws->n_items_static;
    a.item_n = a.region == 0 ? ws->n_items_static : ws->n_items - ws->n_items_static;
}

void attach_far(asc_graph *g, asc_algo algo, RegionArgs &a) {
    if (near_far(g, algo)) {
        a.far_bits = g->ws->far_bits;
        a.thresh = g->ws->ctl + CTL_THRESH;
    }
}

uint32_t grid_for(const Workspace *ws, uint64_t work_items) {
    uint64_t cap = (uint64_t)ws->num_sms * ws->tune.ctas_per_sm;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(cap, work_items));
}

// One wave of bottom-up CTAs (a warp per kBuWords bitmap words per pass).
uint32_t bu_grid(const Workspace *ws, uint64_t nwords) {
    const uint64_t blocks = (nwords + kBuWords * (kBlock / 32) - 1) / (kBuWords * (kBlock / 32));
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(blocks, (uint64_t)ws->num_sms * kBuMinBlocks));
}

// One wave of the item kernels' CTAs, or one per item.
uint32_t item_grid(const Workspace *ws, uint64_t items, uint32_t ctas_per_sm = ASC_PR_ITEM_BLOCKS) {
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(items, (uint64_t)ws->num_sms * ctas_per_sm));
}

uint32_t fill_grid(const Workspace *ws, uint64_t n) {
    uint64_t blocks = (n + kBlock - 1) / kBlock;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(blocks, (uint64_t)ws->num_sms * 8));
}

// The near-far promotion after an expansion (no-ops when the near frontier is
// not empty or the far set is).
void launch_far(asc_graph *g, cudaStream_t s, const RegionArgs &out_args) {
    Workspace *ws = g->ws;
    const uint32_t nwords = (uint32_t)g->V / 32 + 1;
    far_min_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(out_args, nwords, ws->ctl + CTL_MINFAR);
    far_promote_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(out_args, nwords, ws->ctl + CTL_MINFAR,
                                                                 ws->ctl + CTL_THRESH, ws->tune.delta);
}


template <int ALG, int WORDS>
void launch_expand(asc_graph *g, const RegionArgs &a, uint32_t grid) {
    expand_kernel<ALG, WORDS><<<grid, kBlock, 0, g->stream>>>(a);
}

typedef void (*ExpandFn)(asc_graph *, const RegionArgs &, uint32_t);
typedef void (*FusedFn)(cudaStream_t, const FusedArgs &, uint32_t);

template <int ALG, int WORDS>
void launch_fused(cudaStream_t s, const FusedArgs &x, uint32_t grid) {
    expand_fused_kernel<ALG, WORDS><<<grid, kBlock, 0, s>>>(x);
}

// the expansion kernels' WORDS argument for a graph's stored edge layout
int edge_layout(const asc_graph *g) { return g->edge_words == 2 ? 2 : (g->ebits < 32 ? kBitsLayout : 1); }

FusedFn pick_fused(asc_algo algo, int layout) {
    if (algo == ASC_BFS)
        return layout == 2 ? launch_fused<kBFS, 2> : layout == kBitsLayout ? launch_fused<kBFS, kBitsLayout>
                                                                            : launch_fused<kBFS, 1>;
    if (algo == ASC_CC)
        return layout == 2 ? launch_fused<kCC, 2> : layout == kBitsLayout ? launch_fused<kCC, kBitsLayout>
                                                                           : launch_fused<kCC, 1>;
    return layout == 2 ? launch_fused<kSSSP, 2> : layout == kBitsLayout ? launch_fused<kSSSP, kBitsLayout>
                                                                         : launch_fused<kSSSP, 1>;
}

ExpandFn pick_expand(asc_algo algo, int layout) {
    if (algo == ASC_BFS)
        return layout == 2 ? launch_expand<kBFS, 2> : layout == kBitsLayout ? launch_expand<kBFS, kBitsLayout>
                                                                             : launch_expand<kBFS, 1>;
    if (algo == ASC_CC)
        return layout == 2 ? launch_expand<kCC, 2> : layout == kBitsLayout ? launch_expand<kCC, kBitsLayout>
                                                                            : launch_expand<kCC, 1>;
    return layout == 2 ? launch_expand<kSSSP, 2> : layout == kBitsLayout ? launch_expand<kSSSP, kBitsLayout>
                                                                          : launch_expand<kSSSP, 1>;
}

// Per-iteration phase timing with events on the engine's stream.
struct PhaseTimer {
    Workspace *ws;
    bool on;
    size_t used = 0;
    std::vector<int> kind;
    PhaseTimer(Workspace *w, bool enable) : ws(w), on(enable) {}
    asc_status begin(int k) {
        if (!on) return ASC_OK;
        if (ws->phase_events.size() < used + 2) {
            for (int i = 0; i < 64; i++) {
                cudaEvent_t e;
                ASC_CUDA(cudaEventCreate(&e));
                ws->phase_events.push_back(e);
            }
        }
        kind.push_back(k);
        return ASC_OK;
    }
    void record(cudaStream_t s) {
        if (on) cudaEventRecord(ws->phase_events[used++], s);
    }
    asc_status sum(double *ms_by_kind) {
        for (size_t i = 0; i < kind.size(); i++) {
            float ms = 0;
            ASC_CUDA(cudaEventElapsedTime(&ms, ws->phase_events[2 * i], ws->phase_events[2 * i + 1]));
            ms_by_kind[kind[i]] += ms;
        }
        used = 0;
        kind.clear();
        return ASC_OK;
    }
};

// The kernel and grid of a traversal's persistent loop.
typedef void (*TraverseFn)(LoopArgs);
TraverseFn pick_traverse(asc_algo algo, int layout) {
    if (algo == ASC_BFS)
        return layout == 2 ? traverse_kernel<kBFS, 2> : layout == kBitsLayout ? traverse_kernel<kBFS, kBitsLayout>
                                                                               : traverse_kernel<kBFS, 1>;
    if (algo == ASC_CC)
        return layout == 2 ? traverse_kernel<kCC, 2> : layout == kBitsLayout ? traverse_kernel<kCC, kBitsLayout>
                                                                              : traverse_kernel<kCC, 1>;
    return layout == 2 ? traverse_kernel<kSSSP, 2> : layout == kBitsLayout ? traverse_kernel<kSSSP, kBitsLayout>
                                                                            : traverse_kernel<kSSSP, 1>;
}

#ifndef ASC_LOOP_EDGES
#define ASC_LOOP_EDGES 8192
#endif
// CTAs of the persistent loop: all that stay resident, or on a small graph one per
// ASC_LOOP_EDGES edges and vertices, since a barrier costs by its arrivals. Connected
// components read most lists in many iterations: one per 2048. SSSP without thresholds
// does on some graphs: one per 2048 up to 256 CTAs. us at one per 1024 / 2048 / 4096 /
// 8192:
//   BFS   grid of 300 x 300   4826 / 4336 / 4204 / 4201   RMAT scale 16   110 / 88 / 86 / 78
//   SSSP  grid of 300 x 300   5246 / 4899 / 6206 / 8738   RMAT scale 16   196 / 172 / 172 / 191
//   CC    grid of 300 x 300   7655 / 7234 / 9179 / 13805  RMAT scale 16   159 / 139 / 147 / 163
//   CC    path of 4000       38899 / 38902 / 50757 / 61712
// and on 131,072 rings of 8 at 2048 / 4096 / 8192 (912, 768, 384 CTAs): SSSP 131 / 119 /
// 108, CC 193 / 192 / 228 (every vertex at once).
asc_status loop_grid(asc_graph *g, asc_algo algo, TraverseFn fn, uint32_t *grid) {
    Workspace *ws = g->ws;
    int &per_sm = ws->loop_per_sm[algo];
    if (!per_sm) ASC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kBlock, 0));
    const uint64_t resident = (uint64_t)ws->num_sms * std::max(1, std::min(per_sm, (int)ws->tune.ctas_per_sm));
    const uint64_t n = g->E + g->V;
    uint64_t ctas = n / ASC_LOOP_EDGES + 1;
    if (algo == ASC_CC) ctas = n / 2048 + 1;
    else if (algo == ASC_SSSP && !near_far(g, algo)) ctas = std::max(ctas, std::min<uint64_t>(256, n / 2048 + 1));
    *grid = (uint32_t)std::min(resident, ctas);
    return ASC_OK;
}

}  // namespace

// ------------------------------------------- staged dense on-demand passes --
//
// Standard PageRank reads every edge each pass. On a graph opened with staging
// buffers (asc_budget.stage_bytes, part of the device budget), the on-demand
// region is copied each pass in chunks by the copy engine, on a stream of its
// own, into the two device buffers (chunk k into buffer k % 2), while the
// kernels consume the chunk before it; the copy of chunk k + 2 waits only for
// the launch that read chunk k. A chunk is a run of items (merge_plan_kernel), so
// long lists are cut between chunks as between items. The static items are cut
// into as many slices, and launch k runs static slice k with chunk k in one
// grid, so every launch mixes HBM-bound gathers with the staged chunk and the
// copies never wait for the static work. The reference moves its gathered
// partitions into its staging area one at a time with synchronous copies before
// each partition kernel (CalculateOpt.cu:161-178).
struct StageLaunch {
    uint32_t s_begin = 0, s_n = 0;  // static items
    uint32_t c_begin = 0, c_n = 0;  // the chunk's items
    uint64_t w_lo = 0, w_n = 0;     // u32 words the chunk's copy moves, from a 16-byte boundary
};

struct StagePlan {
    std::vector<StageLaunch> launches;  // one per chunk
    uint64_t copy_bytes = 0;         // moved per pass
    uint32_t *d_work = nullptr;      // per launch work cursor
    cudaStream_t copy = nullptr;
    cudaEvent_t copied[2] = {nullptr, nullptr}, consumed[2] = {nullptr, nullptr};
};

void destroy_stage_plan(StagePlan *sp) {
    if (!sp) return;
    if (sp->copy) cudaStreamSynchronize(sp->copy);
    if (sp->d_work) cudaFree(sp->d_work);
    for (int i = 0; i < 2; i++) {
        if (sp->copied[i]) cudaEventDestroy(sp->copied[i]);
        if (sp->consumed[i]) cudaEventDestroy(sp->consumed[i]);
    }
    if (sp->copy) cudaStreamDestroy(sp->copy);
    delete sp;
}

// u32 words of the stored edge array that hold edges [e_lo, e_hi).
void edge_words_of(const asc_graph *g, uint64_t e_lo, uint64_t e_hi, uint64_t &w_lo, uint64_t &w_n) {
    w_lo = w_n = 0;
    if (e_hi <= e_lo) return;
    if (g->edge_words == 2) {
        w_lo = 2 * e_lo;
        w_n = 2 * (e_hi - e_lo);
    } else if (g->ebits == 32) {
        w_lo = e_lo;
        w_n = e_hi - e_lo;
    } else {
        w_lo = (e_lo * g->ebits) >> 5;
        w_n = ((e_hi * g->ebits - 1) >> 5) - w_lo + 1;
    }
}

// The words [w_lo, w_lo + w_n) of the edge array that a copy of edges
// [e_lo, e_hi) moves so that it starts and ends on 16 bytes (or at the end).
void staged_words(const asc_graph *g, uint64_t e_lo, uint64_t e_hi, uint64_t &w_lo, uint64_t &w_n) {
    edge_words_of(g, e_lo, e_hi, w_lo, w_n);
    if (!w_n) return;
    const uint64_t end = std::min<uint64_t>(edge_store_words(g, g->E), (w_lo + w_n + 3) & ~3ull);
    w_lo &= ~3ull;
    w_n = end - w_lo;
}

// The chunks of the graph's on-demand items; *ok false (and no plan) when a
// single item does not fit a staging buffer.
asc_status ensure_stage_plan(asc_graph *g, bool *ok) {
    Workspace *ws = g->ws;
    *ok = false;
    if (!g->stage_words || g->static_edges >= g->E) return ASC_OK;
    if (ws->stage) {
        *ok = true;
        return ASC_OK;
    }
    ASC_TRY(ensure_items(g));
    const uint32_t ns = ws->n_items_static, n = ws->n_items;
    std::vector<uint2> items(n + 1);
    ASC_CUDA(cudaMemcpyAsync(items.data(), ws->items, sizeof(uint2) * items.size(), cudaMemcpyDeviceToHost,
                             g->stream));
    ASC_CUDA(cudaStreamSynchronize(g->stream));
    StagePlan plan;
    for (uint32_t i = ns; i < n;) {
        StageLaunch x;
        x.c_begin = i;
        uint64_t w_lo, w_n;
        for (; i < n; i++) {
            staged_words(g, items[x.c_begin].y, items[i + 1].y, w_lo, w_n);
            if (w_n > g->stage_words) break;
            x.w_lo = w_lo;
            x.w_n = w_n;
        }
        x.c_n = i - x.c_begin;
        if (!x.c_n) return ASC_OK;
        plan.copy_bytes += 4 * x.w_n;
        plan.launches.push_back(x);
    }
    const uint64_t L = plan.launches.size();
    for (uint64_t k = 0; k < L; k++) {
        StageLaunch &x = plan.launches[k];
        x.s_begin = (uint32_t)(k * ns / L);
        x.s_n = (uint32_t)((k + 1) * ns / L) - x.s_begin;
    }
    StagePlan *sp = new StagePlan(plan);
    asc_status st = ASC_OK;
    auto cu = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && st == ASC_OK) st = cuda_fail(e, what, __FILE__, __LINE__);
    };
    cu(cudaMalloc(&sp->d_work, 4 * L), "cudaMalloc(stage cursors)");
    if (st == ASC_OK) cu(cudaStreamCreateWithFlags(&sp->copy, cudaStreamNonBlocking), "cudaStreamCreate");
    for (int i = 0; i < 2 && st == ASC_OK; i++) {
        cu(cudaEventCreateWithFlags(&sp->copied[i], cudaEventDisableTiming), "cudaEventCreate");
        cu(cudaEventCreateWithFlags(&sp->consumed[i], cudaEventDisableTiming), "cudaEventCreate");
    }
    if (st != ASC_OK) {
        destroy_stage_plan(sp);
        return st;
    }
    ws->stage = sp;
    *ok = true;
    return ASC_OK;
}

// Whole-partition comparison engine (ASC_RUN_PARTITION_COPY), the reference's
// baseline of bfs.cu:6-168 / gpu_kernels.cu:302-519: the on-demand region in
// partitions of one staging buffer, cut at vertex boundaries only; each
// iteration copies every partition that holds a frontier vertex, whole, and
// expands that partition's frontier vertices from the copy.
struct Partition {
    uint32_t v_lo = 0, v_hi = 0;  // vertices
    uint64_t w_lo = 0, w_n = 0;   // u32 words of their lists
};

struct PartPlan {
    std::vector<Partition> parts;
    uint32_t *d_ranges = nullptr;    // per partition: tile range
    uint32_t *d_flags = nullptr;     // per partition: holds a frontier vertex this iteration
    uint32_t *h_flags = nullptr;     // page-locked mirror
    uint32_t *d_cnt = nullptr;       // per partition, 8 words: an id-order walk of its range, no segments
    uint32_t *d_work = nullptr;      // per partition work cursor
    cudaStream_t copy = nullptr;
    cudaEvent_t copied[2] = {nullptr, nullptr}, consumed[2] = {nullptr, nullptr};
};

void destroy_part_plan(PartPlan *pp) {
    if (!pp) return;
    if (pp->copy) cudaStreamSynchronize(pp->copy);
    for (void *q : {(void *)pp->d_ranges, (void *)pp->d_flags, (void *)pp->d_cnt, (void *)pp->d_work})
        if (q) cudaFree(q);
    if (pp->h_flags) cudaFreeHost(pp->h_flags);
    for (int i = 0; i < 2; i++) {
        if (pp->copied[i]) cudaEventDestroy(pp->copied[i]);
        if (pp->consumed[i]) cudaEventDestroy(pp->consumed[i]);
    }
    if (pp->copy) cudaStreamDestroy(pp->copy);
    delete pp;
}

asc_status ensure_part_plan(asc_graph *g) {
    Workspace *ws = g->ws;
    if (ws->part) return ASC_OK;
    if (!g->stage_words)
        return fail(ASC_ERR_INVALID, "the partition-copy engine needs staging buffers (asc_budget.stage_bytes)");
    const uint32_t V = (uint32_t)g->V, S = g->static_vertices;
    std::vector<Partition> parts(1);
    const uint64_t cap = g->stage_words;
    parts[0].v_lo = parts[0].v_hi = S;
    for (uint32_t v = S; v < V; v++) {
        uint64_t w_lo, w_n;
        edge_words_of(g, g->h_ptr[parts.back().v_lo], g->h_ptr[v + 1], w_lo, w_n);
        if (w_n > cap) {
            Partition next;
            next.v_lo = v;
            edge_words_of(g, g->h_ptr[v], g->h_ptr[v + 1], w_lo, w_n);
            if (w_n > cap)
                return fail(ASC_ERR_BUDGET, "an adjacency list is longer than a partition (%llu words)",
                            (unsigned long long)cap);
            parts.push_back(next);
        }
        parts.back().v_hi = v + 1;
        parts.back().w_lo = w_lo;
        parts.back().w_n = w_n;
    }
    PartPlan *pp = new PartPlan();
    const size_t n = parts.size();
    std::vector<uint32_t> ranges(2 * n), cnt(8 * n, 0);
    for (size_t k = 0; k < n; k++) {
        ranges[2 * k] = parts[k].v_lo;
        ranges[2 * k + 1] = parts[k].v_hi;
        cnt[8 * k + 7] = 1;  // with dense_div at its maximum: walk the range in id order
    }
    pp->parts = std::move(parts);
    asc_status st = ASC_OK;
    auto cu = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && st == ASC_OK) st = cuda_fail(e, what, __FILE__, __LINE__);
    };
    cu(cudaMalloc(&pp->d_ranges, 8 * n), "cudaMalloc(partition ranges)");
    cu(cudaMalloc(&pp->d_flags, 4 * n), "cudaMalloc(partition flags)");
    cu(cudaMalloc(&pp->d_cnt, 32 * n), "cudaMalloc(partition counts)");
    cu(cudaMalloc(&pp->d_work, 4 * n), "cudaMalloc(partition cursors)");
    cu(cudaHostAlloc((void **)&pp->h_flags, 4 * n, cudaHostAllocDefault), "cudaHostAlloc(partition flags)");
    if (st == ASC_OK) cu(cudaMemcpy(pp->d_ranges, ranges.data(), 8 * n, cudaMemcpyHostToDevice), "cudaMemcpy");
    if (st == ASC_OK) cu(cudaMemcpy(pp->d_cnt, cnt.data(), 32 * n, cudaMemcpyHostToDevice), "cudaMemcpy");
    if (st == ASC_OK) cu(cudaStreamCreateWithFlags(&pp->copy, cudaStreamNonBlocking), "cudaStreamCreate");
    for (int i = 0; i < 2 && st == ASC_OK; i++) {
        cu(cudaEventCreateWithFlags(&pp->copied[i], cudaEventDisableTiming), "cudaEventCreate");
        cu(cudaEventCreateWithFlags(&pp->consumed[i], cudaEventDisableTiming), "cudaEventCreate");
    }
    if (st != ASC_OK) {
        destroy_part_plan(pp);
        return st;
    }
    ws->part = pp;
    return ASC_OK;
}

// One CTA per partition (grid-stride): whether its tile range holds a vertex
// of this iteration's frontier.
__global__ void part_active_kernel(const uint32_t *bitmap_in, const uint32_t *ranges, uint32_t n,
                                   uint32_t *flags) {
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        const uint32_t lo = ranges[2 * k], hi = ranges[2 * k + 1];
        uint32_t any = 0;
        for (uint32_t u0 = (lo & ~31u) + 32 * threadIdx.x; u0 < hi; u0 += 32 * blockDim.x) {
            uint32_t w = bitmap_in[u0 >> 5];
            if (u0 < lo) w &= 0xffffffffu << (lo - u0);
            if (hi - u0 < 32u) w &= (1u << (hi - u0)) - 1u;
            any |= w;
        }
        any = __syncthreads_or(any != 0);
        if (threadIdx.x == 0) flags[k] = any;
    }
}

// Launch k's slices: static items in place and the chunk, whose copy goes to the
// copy stream once the launch that last read the same buffer is done; the
// compute stream s waits for it.
asc_status stage_chunk(asc_graph *g, StagePlan *sp, uint32_t k, cudaStream_t s, PrSlice sl[2]) {
    const StageLaunch &x = sp->launches[k];
    sl[0] = pr_slice(g, 0);
    sl[0].begin = x.s_begin;
    sl[0].n = x.s_n;
    sl[1].begin = x.c_begin;
    sl[1].n = x.c_n;
    sl[1].edges = g->d_stage[k & 1];
    sl[1].edge_words = 0;
    if (!x.w_n) return ASC_OK;  // rows without edges
    ASC_CUDA(cudaStreamWaitEvent(sp->copy, sp->consumed[k & 1], 0));
    ASC_CUDA(cudaMemcpyAsync(g->d_stage[k & 1], g->h_edges + x.w_lo, 4 * x.w_n, cudaMemcpyHostToDevice, sp->copy));
    ASC_CUDA(cudaEventRecord(sp->copied[k & 1], sp->copy));
    ASC_CUDA(cudaStreamWaitEvent(s, sp->copied[k & 1], 0));
    // indexed by global edge offset: the buffer less the chunk's first word
    sl[1].edges = (const uint32_t *)((uintptr_t)g->d_stage[k & 1] - 4 * (uintptr_t)x.w_lo);
    sl[1].edge_words = x.w_lo + x.w_n;
    return ASC_OK;
}

asc_status stage_release(StagePlan *sp, uint32_t k, cudaStream_t s) {
    if (sp->launches[k].w_n) ASC_CUDA(cudaEventRecord(sp->consumed[k & 1], s));
    return ASC_OK;
}

void free_ws_buffers(Workspace *ws) {
    for (void *p : {(void *)ws->val, (void *)ws->visited, (void *)ws->huge_bits, (void *)ws->far_bits,
                    (void *)ws->frag_counts,
                    (void *)ws->bitmap[0],
                    (void *)ws->bitmap[1],
                    (void *)ws->queue[0],
                    (void *)ws->queue[1],
                    (void *)ws->segs[0], (void *)ws->segs[1], (void *)ws->ctl, ws->pr_rank,
                    ws->pr_contrib[0], ws->pr_contrib[1], ws->pr_sum, (void *)ws->items, (void *)ws->pr_hot, (void *)ws->in_ptr, (void *)ws->in_edges,
                    (void *)ws->in_none})
        if (p) cudaFree(p);
    if (ws->h_ctl) cudaFreeHost(ws->h_ctl);
    for (void *p : {(void *)ws->g_stage, (void *)ws->g_items})
        if (p) cudaFree(p);
    for (void *p : {(void *)ws->h_stage, (void *)ws->h_items, (void *)ws->h_list, (void *)ws->h_segs})
        if (p) cudaFreeHost(p);
    for (auto e : ws->ev)
        if (e) cudaEventDestroy(e);
    for (auto e : ws->phase_events) cudaEventDestroy(e);
    for (auto e : ws->pass_ev)
        if (e) cudaEventDestroy(e);
    destroy_stage_plan(ws->stage);
    ws->stage = nullptr;
    destroy_part_plan(ws->part);
    ws->part = nullptr;
}

void free_workspace(asc_graph *g) {
    Workspace *ws = g->ws;
    if (!ws) return;
    for (auto &b : ws->batch)
        if (b) {
            batch_destroy(b);
            b = nullptr;
        }
    free_ws_buffers(ws);
    delete ws;
    g->ws = nullptr;
}

asc_status run_traversal_impl(asc_graph *g, asc_algo algo, uint32_t source, const asc_params &p, void *out,
                              asc_stats *st);

uint64_t fragment_count(const asc_graph *g) { return (g->E + 4095) / 4096; }

asc_status run_traversal(asc_graph *g, asc_algo algo, uint32_t source, const asc_params &p, void *out,
                         asc_stats *st) {
    ASC_TRY(ensure_workspace(g));
    Workspace *ws = g->ws;
    if (p.flags & ASC_RUN_FRAGMENT_COUNTS) {
        if (!ws->frag_counts) {
            const size_t bytes = 8 * std::max<uint64_t>(1, fragment_count(g));
            ASC_CUDA(cudaMalloc(&ws->frag_counts, bytes));
            ASC_CUDA(cudaMemsetAsync(ws->frag_counts, 0, bytes, g->stream));
            ws->device_bytes += bytes;
        }
        ws->frag_active = ws->frag_counts;
    }
    // the gather engine expands the on-demand region from its frontier list
    const uint32_t div = ws->tune.dense_div;
    if (p.flags & ASC_RUN_GATHER_COPY) ws->tune.dense_div = 0;
    const asc_status rc = run_traversal_impl(g, algo, source, p, out, st);
    ws->tune.dense_div = div;
    ws->frag_active = nullptr;
    return rc;
}

typedef void (*StagedFn)(cudaStream_t, const StagedArgs &, uint32_t);

template <int ALG, int WORDS>
void launch_staged(cudaStream_t s, const StagedArgs &x, uint32_t grid) {
    expand_staged_kernel<ALG, WORDS><<<grid, kBlock, 0, s>>>(x);
}

StagedFn pick_staged(asc_algo algo, bool pairs) {
    if (algo == ASC_BFS) return pairs ? launch_staged<kBFS, 2> : launch_staged<kBFS, 1>;
    if (algo == ASC_CC) return pairs ? launch_staged<kCC, 2> : launch_staged<kCC, 1>;
    return pairs ? launch_staged<kSSSP, 2> : launch_staged<kSSSP, 1>;
}

// Host side of the gather-and-copy engine for one iteration: the on-demand
// list and segments come back to the host, host threads gather their edges
// (decoding the stored layout) into page-locked staging in parts of at most
// g_cap edges, and each part is copied over and expanded before the next.
asc_status gather_ondemand(asc_graph *g, asc_algo algo, int parity, const uint32_t *cnt, cudaEvent_t lists_ready,
                           uint32_t &launches) {
    Workspace *ws = g->ws;
    cudaStream_t s = g->stream;
    const uint32_t n_list = cnt[1], n_seg = cnt[3];
    ASC_CUDA(cudaEventSynchronize(lists_ready));
    if (!n_list && !n_seg) return ASC_OK;
    const uint32_t words = g->edge_words;
    const uint32_t seg_len = ws->tune.segment_edges;
    struct Item { uint32_t u; uint64_t b; uint32_t len, first; };
    std::vector<Item> items;
    items.reserve((size_t)n_list + n_seg);
    for (uint32_t i = 0; i < n_list; i++) {
        const uint32_t u = ws->h_list[i];
        items.push_back({u, g->h_ptr[u], g->h_ptr[u + 1] - g->h_ptr[u], 1u});
    }
    for (uint32_t i = 0; i < n_seg; i++) {
        const uint32_t u = (uint32_t)(ws->h_segs[i] >> 32), k = (uint32_t)ws->h_segs[i];
        const uint64_t b = (uint64_t)g->h_ptr[u] + (uint64_t)k * seg_len;
        const uint64_t e = std::min<uint64_t>(g->h_ptr[u + 1], b + seg_len);
        items.push_back({u, b, (uint32_t)(e - b), k == 0 ? 1u : 0u});
    }
    const uint32_t *he = g->h_edges;
    const uint32_t eb = g->ebits;
    auto word_at = [&](uint64_t idx) -> uint32_t {
        if (words == 2 || eb == 32) return he[idx];
        const uint64_t bit = idx * eb;
        const uint32_t sh = (uint32_t)(bit & 31);
        uint32_t x = he[bit >> 5] >> sh;
        if (sh + eb > 32) x |= he[(bit >> 5) + 1] << (32 - sh);
        return x & ((1u << eb) - 1u);
    };
    const unsigned hw = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    const StagedFn staged = pick_staged(algo, words == 2);
    size_t i0 = 0;
    while (i0 < items.size()) {
        // one part: items whose edges fit the staging buffer
        uint64_t tot = 0;
        size_t i1 = i0;
        while (i1 < items.size() && i1 - i0 < ws->g_cap && tot + items[i1].len <= ws->g_cap) tot += items[i1++].len;
        const size_t n = i1 - i0;
        std::vector<uint64_t> off(n + 1, 0);
        for (size_t k = 0; k < n; k++) off[k + 1] = off[k] + items[i0 + k].len;
        auto work = [&](unsigned t) {
            for (size_t k = t; k < n; k += hw) {
                const Item &it = items[i0 + k];
                uint32_t *dst = ws->h_stage + off[k] * words;
                if (words == 2) memcpy(dst, he + 2 * it.b, 8ull * it.len);
                else for (uint32_t j = 0; j < it.len; j++) dst[j] = word_at(it.b + j);
                uint32_t *q = ws->h_items + 4 * k;
                q[0] = it.u;
                q[1] = (uint32_t)off[k];
                q[2] = it.len;
                q[3] = it.first;
            }
        };
        std::vector<std::thread> th;
        for (unsigned t = 1; t < hw; t++) th.emplace_back(work, t);
        work(0);
        for (auto &x : th) x.join();
        ASC_CUDA(cudaMemcpyAsync(ws->g_stage, ws->h_stage, 4ull * words * tot, cudaMemcpyHostToDevice, s));
        ASC_CUDA(cudaMemcpyAsync(ws->g_items, ws->h_items, 16ull * n, cudaMemcpyHostToDevice, s));
        StagedArgs x;
        x.a = region_args(g, parity, 1, false);
        attach_far(g, algo, x.a);
        x.stage = ws->g_stage;
        x.items = ws->g_items;
        x.n_items = (uint32_t)n;
        staged(s, x, fill_grid(ws, 32ull * n));
        launches++;
        ASC_CUDA(cudaGetLastError());
        // the staging buffers are reused by the next part
        ASC_CUDA(cudaStreamSynchronize(s));
        i0 = i1;
    }
    return ASC_OK;
}

asc_status ensure_gather_buffers(asc_graph *g) {
    Workspace *ws = g->ws;
    if (ws->g_stage) return ASC_OK;
    const uint64_t od = g->E - std::min<uint64_t>(g->E, g->h_ptr[g->static_vertices]);
    // a part must hold the longest item: a list up to huge_degree edges or a segment
    const uint64_t need = std::max<uint64_t>(ws->tune.huge_degree, ws->tune.segment_edges);
    ws->g_cap = std::max<uint64_t>(need, std::min<uint64_t>(std::max<uint64_t>(od, 1), 1ull << 25));
    const uint64_t words = g->edge_words;
    ASC_CUDA(cudaMalloc(&ws->g_stage, 4 * words * ws->g_cap));
    ASC_CUDA(cudaMalloc(&ws->g_items, 16 * ws->g_cap));
    ASC_CUDA(cudaHostAlloc(&ws->h_stage, 4 * words * ws->g_cap, cudaHostAllocDefault));
    ASC_CUDA(cudaHostAlloc(&ws->h_items, 16 * ws->g_cap, cudaHostAllocDefault));
    ASC_CUDA(cudaHostAlloc(&ws->h_list, 4 * (g->V + 1), cudaHostAllocDefault));
    ASC_CUDA(cudaHostAlloc(&ws->h_segs, 8 * (ws->segcap_ondemand + 1), cudaHostAllocDefault));
    return ASC_OK;
}

// ------------------------------------------- in-edges of a CSR graph -------
//
// Built on the device on the graph's first BFS: in-degrees counted over the merge
// items, scanned to offsets, then one pass over all edges for every run of lists
// that fits a queue of the workspace (V entries; nothing else is allocated on the
// device), which scatters the run's sources, moves the best candidate of each list
// to its front and packs the run into page-locked memory. On host threads this
// took 4.0 s for the 268 M edges of RMAT scale 24.
//
// The first in-edge of a list is the source with the most out-edges among the first
// kHeadSample that arrived: the one most likely to be in a large frontier. Of the 7% of
// vertices whose smallest-id source was no parent in the large step of a BFS on RMAT
// scale 21, 24,200 went on to read host memory; with this choice 3,744 do. The others
// follow in the order in which the scatter's atomics came, which differs from one build
// to the next (host-built lists are sorted): the levels do not depend on it, the number
// of in-edges that a step reads does.
namespace {

struct InEdgeArgs {
    const uint2 *items;
    PrSlice sl[2];
    const uint32_t *ptr;
    uint32_t *cnt;           // in-degrees, then cursors
    uint32_t *raw;           // the run's sources by list
    uint32_t V, ebits, wbits;
    uint32_t lo, hi, base;   // the run: lists [lo, hi), the first starts at base
};

template <bool COUNT>
__global__ void __launch_bounds__(kBlock, 6) in_edges_kernel(InEdgeArgs p) {
    __shared__ PrItemSmem<float> sm;
    const int lane = threadIdx.x & 31;
    const uint32_t total = p.sl[0].n + p.sl[1].n;
    const uint32_t eb = p.ebits, mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
    uint32_t *marks = sm.marks[0];
    for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
        bool od;
        const uint32_t it = pr_slice_item(p.sl, w, od);
        const uint2 a = p.items[it], b = p.items[it + 1];
        const uint32_t r0 = a.x, e0 = a.y, nr = b.x - a.x, ne = b.y - a.y;
        uint32_t nq;
        if (threadIdx.x < kItem / 32) marks[threadIdx.x] = 0;
        const uint32_t bit0 = stage_words(p.sl[od].edges, p.sl[od].edge_words, e0, ne, eb, sm.pool, nq);
        __syncthreads();
        if (!COUNT) {
            pr_mark_rows<float>(p.ptr, r0, e0, nr, sm, marks);
            __syncthreads();
        }
        const uint32_t x0 = threadIdx.x * kVt, xw = x0 - lane * kVt;
        if (xw < ne) {
            uint32_t ends = 0, open = 0, row = 0;
            if (!COUNT) {
                ends = (marks[x0 >> 5] >> (x0 & 31)) & ((1u << kVt) - 1u);
                const unsigned ended = __ballot_sync(kFull, ends != 0);
                const uint32_t first = ends ? sm.row_at[x0 + __ffs((int)ends) - 1] : nr;
                const unsigned above = lane < 31 ? ended & (0xffffffffu << (lane + 1)) : 0u;
                const uint32_t from_lane = __shfl_sync(kFull, first, above ? __ffs((int)above) - 1 : lane);
                const uint32_t after = pr_next_row(marks, sm.row_at, xw + 32 * kVt, nr);
                open = above ? from_lane : after;
                row = ends ? first : open;
            }
#pragma unroll
            for (int k = 0; k < kVt; k++) {
                if (x0 + k < ne) {
                    const uint32_t v = staged_word(sm.pool, bit0 + (x0 + k) * eb, mask) >> p.wbits;
                    if (!ASC_BAD(v >= p.V, 24, v)) {
                        if (COUNT) atomicAdd(&p.cnt[v], 1u);
                        else if (v >= p.lo && v < p.hi) p.raw[atomicAdd(&p.cnt[v], 1u) - p.base] = r0 + row;
                    }
                }
                if (!COUNT && ((ends >> k) & 1u)) {
                    const uint32_t rest = ends >> k >> 1;
                    row = rest ? (uint32_t)sm.row_at[x0 + k + __ffs((int)rest)] : open;
                }
            }
        }
        __syncthreads();
    }
}

// Exclusive scan of cnt[V] in blocks of kItem: block sums, their scan, the
// offsets (also left in cnt as the scatter's cursors).
__global__ void scan_sums_kernel(const uint32_t *cnt, uint32_t V, uint32_t *sums) {
    __shared__ uint32_t warp[kWarps + 1];
    uint32_t x = 0, total;
    for (int k = 0; k < kVt; k++) {
        const uint64_t v = (uint64_t)blockIdx.x * kItem + k * kBlock + threadIdx.x;
        if (v < V) x += cnt[v];
    }
    block_excl_scan(x, total, warp);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void scan_block_sums_kernel(uint32_t *sums, uint32_t n) {
    __shared__ uint32_t warp[kWarps + 1];
    uint32_t run = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += kBlock) {
        const uint32_t i = i0 + threadIdx.x, x = i < n ? sums[i] : 0;
        uint32_t total;
        const uint32_t before = block_excl_scan(x, total, warp);
        if (i < n) sums[i] = run + before;
        run += total;
        __syncthreads();
    }
}

__global__ void scan_offsets_kernel(uint32_t *cnt, uint32_t V, const uint32_t *sums, uint32_t E, uint32_t *in_ptr,
                                    uint32_t *in_none) {
    __shared__ uint32_t warp[kWarps + 1];
    const uint64_t v0 = (uint64_t)blockIdx.x * kItem + threadIdx.x * kVt;
    uint32_t c[kVt], x = 0, total;
#pragma unroll
    for (int k = 0; k < kVt; k++) {
        c[k] = v0 + k < V ? cnt[v0 + k] : 0;
        x += c[k];
    }
    uint32_t run = sums[blockIdx.x] + block_excl_scan(x, total, warp);
    uint32_t none = 0;
#pragma unroll
    for (int k = 0; k < kVt; k++) {
        if (v0 + k < V) in_ptr[v0 + k] = cnt[v0 + k] = run;
        if (v0 + k >= V || !c[k]) none |= 1u << k;
        run += c[k];
    }
    // four threads' bytes are a word of the bitmap of vertices without in-edges
    // (bits past V set: nothing to look for there)
    none <<= 8 * (threadIdx.x & 3);
    none |= __shfl_xor_sync(kFull, none, 1);
    none |= __shfl_xor_sync(kFull, none, 2);
    if ((threadIdx.x & 3) == 0 && v0 / 32 < V / 32 + 2) in_none[v0 / 32] = none;
    if (blockIdx.x == 0 && threadIdx.x == 0) in_ptr[V] = E;
}

// A warp per list of the run: the source with the most out-edges among its first
// kHeadSample goes to the front, and to heads[v] (a vertex without in-edges: itself).
constexpr uint32_t kHeadSample = 4096;
__global__ void in_heads_kernel(InEdgeArgs p, const uint32_t *in_ptr, uint32_t *heads) {
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * kWarps;
    for (uint64_t v = (uint64_t)p.lo + blockIdx.x * kWarps + (threadIdx.x >> 5); v < p.hi; v += warps) {
        const uint32_t b = in_ptr[v] - p.base, n = in_ptr[v + 1] - in_ptr[v];
        unsigned long long best = 0;  // out-degree, then the smaller id
        uint32_t at = 0;
        for (uint32_t i = lane; i < min(n, kHeadSample); i += 32) {
            const uint32_t u = p.raw[b + i];
            const unsigned long long key = ((unsigned long long)(p.ptr[u + 1] - p.ptr[u]) << 32) | (0xffffffffu - u);
            if (key > best) {
                best = key;
                at = i;
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const unsigned long long k2 = __shfl_xor_sync(kFull, best, d);
            const uint32_t a2 = __shfl_xor_sync(kFull, at, d);
            if (k2 > best || (k2 == best && a2 < at)) {
                best = k2;
                at = a2;
            }
        }
        if (lane == 0) {
            if (n) {
                const uint32_t u = p.raw[b + at];
                p.raw[b + at] = p.raw[b];
                p.raw[b] = u;
                heads[v] = u;
            } else {
                heads[v] = (uint32_t)v;
            }
        }
    }
}

// Packs src[0, n) (words first .. first + n - 1 of a stream of eb bits each) into
// out. The last word, when words of a later call share it, goes to *carry_out,
// and the first takes what an earlier call left in *carry_in.
__global__ void pack_stream_kernel(const uint32_t *src, uint64_t first, uint64_t n, uint32_t eb, uint32_t *out,
                                   const uint32_t *carry_in, uint32_t *carry_out, bool last) {
    const uint64_t bit_lo = first * eb, bit_hi = (first + n) * eb;
    const uint64_t w_lo = bit_lo >> 5, w_hi = (bit_hi + 31) >> 5;
    for (uint64_t w = w_lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < w_hi;
         w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b0 = 32 * w;
        uint32_t x = w == w_lo && (bit_lo & 31) ? *carry_in : 0u;
        for (uint64_t i = max(first, b0 / eb); i < first + n && i * eb < b0 + 32; i++) {
            const uint32_t y = src[i - first];
            x |= i * eb >= b0 ? y << (i * eb - b0) : y >> (b0 - i * eb);
        }
        if (w == w_hi - 1 && (bit_hi & 31) && !last) *carry_out = x;
        else out[w] = x;
    }
}

// *done false (and nothing kept) where a list is longer than a queue or the runs
// would be many: the host builds those.
asc_status in_edges_on_device(asc_graph *g, bool *done) {
    Workspace *ws = g->ws;
    cudaStream_t s = g->stream;
    const uint64_t V = g->V, E = g->E;
    constexpr uint64_t kMaxRuns = 64;
    *done = false;
    if (!E || E / V >= kMaxRuns) return ASC_OK;
    ASC_TRY(ensure_items(g));
    InEdgeArgs p;
    memset(&p, 0, sizeof(p));
    p.items = ws->items;
    p.sl[0] = pr_slice(g, 0);
    p.sl[1] = pr_slice(g, 1);
    p.ptr = g->d_ptr;
    p.cnt = ws->val;
    p.raw = ws->queue[0];
    p.V = (uint32_t)V;
    p.ebits = g->edge_words == 2 ? 64 : g->ebits;
    p.wbits = g->wbits;
    const uint32_t blocks = (uint32_t)((V + 63 + kItem) / kItem), grid = item_grid(ws, ws->n_items, 6);
    uint32_t *heads = ws->queue[1], *carry = ws->ctl + CTL_BARRIER + 1;
    ASC_CUDA(cudaMemsetAsync(p.cnt, 0, 4 * V, s));
    ASC_CUDA(cudaMemsetAsync(carry, 0, 8, s));
    in_edges_kernel<true><<<grid, kBlock, 0, s>>>(p);
    // the block sums fit a queue: V / kItem + 2 words; graphs too small for that go to the host
    if (blocks > V) return ASC_OK;
    scan_sums_kernel<<<blocks, kBlock, 0, s>>>(p.cnt, p.V, heads);
    scan_block_sums_kernel<<<1, kBlock, 0, s>>>(heads, blocks);
    scan_offsets_kernel<<<blocks, kBlock, 0, s>>>(p.cnt, p.V, heads, (uint32_t)E, ws->in_ptr, ws->in_none);
    ASC_CUDA(cudaGetLastError());
    std::unique_ptr<uint32_t[]> h_ptr(new (std::nothrow) uint32_t[V + 1]);
    std::unique_ptr<uint32_t[]> none(new (std::nothrow) uint32_t[V / 32 + 2]);
    if (!h_ptr || !none) return fail(ASC_ERR_NOMEM, "in-edge offsets: %llu vertices", (unsigned long long)V);
    const uint32_t *in_ptr = h_ptr.get();
    ASC_CUDA(cudaMemcpyAsync(h_ptr.get(), ws->in_ptr, 4 * (V + 1), cudaMemcpyDeviceToHost, s));
    ASC_CUDA(cudaStreamSynchronize(s));
    uint32_t cuts[2 * kMaxRuns + 1] = {0}, runs = 0;  // runs of lists of at most V entries
    while (cuts[runs] < V) {
        const uint32_t lo = cuts[runs];
        const uint32_t hi = (uint32_t)(std::upper_bound(in_ptr + lo, in_ptr + V + 1, in_ptr[lo] + V,
                                                        [](uint64_t x, uint32_t y) { return x < y; }) -
                                       in_ptr) - 1;
        if (hi <= lo || runs == 2 * kMaxRuns) return ASC_OK;
        cuts[++runs] = hi;
    }
    const uint32_t bits = g->in_ebits;
    const uint64_t words = in_edge_words(g);
    uint32_t *packed = nullptr;
    if (cudaHostAlloc((void **)&packed, 4 * ((words + 3) & ~3ull), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return fail(ASC_ERR_NOMEM, "cudaHostAlloc of %llu bytes failed", (unsigned long long)(4 * words));
    }
    void *dp = nullptr;
    cudaError_t e = cudaHostGetDevicePointer(&dp, packed, 0);
    const uint32_t fill = fill_grid(ws, ~0ull >> 32);
    for (uint32_t k = 0; e == cudaSuccess && k < runs; k++) {
        p.lo = cuts[k];
        p.hi = cuts[k + 1];
        p.base = in_ptr[p.lo];
        const uint64_t n = in_ptr[p.hi] - p.base;
        const bool last = k + 1 == runs;
        in_edges_kernel<false><<<grid, kBlock, 0, s>>>(p);
        in_heads_kernel<<<fill, kBlock, 0, s>>>(p, ws->in_ptr, heads);
        if (n) pack_stream_kernel<<<fill, kBlock, 0, s>>>(p.raw, p.base, n, bits, (uint32_t *)dp, carry + (k & 1),
                                                           carry + (1 - (k & 1)), last);
        else e = cudaMemcpyAsync(carry + (1 - (k & 1)), carry + (k & 1), 4, cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess && g->d_in_heads && !g->in_heads_ready) {
        e = cudaMemsetAsync(g->d_in_heads, 0, 4 * g->in_head_words, s);
        pack_stream_kernel<<<fill, kBlock, 0, s>>>(heads, 0, V, bits, g->d_in_heads, carry, carry, true);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(none.get(), ws->in_none, 4 * (V / 32 + 2), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaFreeHost(packed);
        return cuda_fail(e, "in-edges", __FILE__, __LINE__);
    }
    if (bits < 32) packed[words - 1] = 0;  // the padding word
    g->h_in_ptr = h_ptr.release();
    g->h_in_none = none.release();
    g->h_in_edges = packed;
    g->d_host_in_edges = (const uint32_t *)dp;
    if (g->d_in_heads) g->in_heads_ready = true;
    *done = true;
    return ASC_OK;
}

}  // namespace

// In-edge offsets on the device for bottom-up BFS steps, built on the
// graph's first BFS. The in-edges stay in pinned host memory, read in place,
// unless the graph has no cap (every out-edge resident): then they are
// resident too.
asc_status ensure_in_ptr(asc_graph *g) {
    Workspace *ws = g->ws;
    if (ws->in_ptr) return ASC_OK;
    const uint64_t nw = g->V / 32 + 2;
    ASC_CUDA(cudaMalloc(&ws->in_ptr, 4 * (g->V + 1)));
    ws->device_bytes += 4 * (g->V + 1);
    ASC_CUDA(cudaMalloc(&ws->in_none, 4 * nw));
    ws->device_bytes += 4 * nw;
    bool on_device = false;
    asc_status st = g->h_in_edges ? ASC_OK : in_edges_on_device(g, &on_device);
    if (st == ASC_OK && !on_device) {
        if (!g->h_in_edges) st = build_in_edges(g);
        if (st == ASC_OK && !g->h_in_none) {
            uint32_t *none = new uint32_t[nw]();
            for (uint64_t v = 0; v < 32 * nw; v++)
                if (v >= g->V || g->h_in_ptr[v + 1] == g->h_in_ptr[v]) none[v >> 5] |= 1u << (v & 31);
            g->h_in_none = none;
        }
        // the graph's host copies: a server that freed the state of an idle graph uploads them again
        auto up = [&](void *to, const void *from, size_t n) {
            if (st != ASC_OK) return;
            const cudaError_t e = cudaMemcpy(to, from, n, cudaMemcpyHostToDevice);
            if (e != cudaSuccess) st = cuda_fail(e, "in-edge offsets", __FILE__, __LINE__);
        };
        up(ws->in_ptr, g->h_in_ptr, 4 * (g->V + 1));
        up(ws->in_none, g->h_in_none, 4 * nw);
    }
    if (st != ASC_OK) {  // in_ptr marks the state as complete
        cudaFree(ws->in_ptr);
        cudaFree(ws->in_none);
        ws->in_ptr = ws->in_none = nullptr;
        ws->device_bytes -= 4 * (g->V + 1) + 4 * nw;
        return st;
    }
    if (g->static_edges >= g->E) {
        const uint64_t words = in_edge_words(g);
        ASC_CUDA(cudaMalloc(&ws->in_edges, 4 * ((words + 3) & ~3ull)));
        ASC_CUDA(cudaMemcpy(ws->in_edges, g->h_in_edges, 4 * words, cudaMemcpyHostToDevice));
        ws->device_bytes += 4 * words;
    }
    return ASC_OK;
}

asc_status run_traversal_impl(asc_graph *g, asc_algo algo, uint32_t source, const asc_params &p, void *out,
                              asc_stats *st) {
    Workspace *ws = g->ws;
    const uint32_t V = (uint32_t)g->V;
    cudaStream_t s = g->stream;
    const bool all = algo == ASC_CC;
    uint32_t launches = 0;
    PhaseTimer pt(ws, (p.flags & ASC_RUN_PHASE_TIMING) != 0);
    // bottom-up steps: BFS on a CSR graph, in the persistent loop or the host
    // loop (the per-region timing, fragment counting and gather-and-copy runs
    // measure the top-down expansion alone)
    ws->bu_active = algo == ASC_BFS && ws->tune.bu_div && !g->is_csc &&
                    !(p.flags & (ASC_RUN_FRAGMENT_COUNTS | ASC_RUN_GATHER_COPY | ASC_RUN_PARTITION_COPY));
    if (ws->bu_active) ASC_TRY(ensure_in_ptr(g));
    ExpandFn expand = pick_expand(algo, edge_layout(g));
    FusedFn fused = pick_fused(algo, edge_layout(g));

    const int64_t cap = p.max_iterations > 0 ? p.max_iterations : (int64_t)4 * V + 64;
    const bool gather = (p.flags & ASC_RUN_GATHER_COPY) != 0;
    if (gather) ASC_TRY(ensure_gather_buffers(g));
    const bool part = !gather && (p.flags & ASC_RUN_PARTITION_COPY) != 0;
    if (part) ASC_TRY(ensure_part_plan(g));
    const bool device_loop = !(p.flags & (ASC_RUN_PHASE_TIMING | ASC_RUN_HOST_LOOP | ASC_RUN_FRAGMENT_COUNTS |
                                          ASC_RUN_GATHER_COPY | ASC_RUN_PARTITION_COPY));
    // regions walked in id order go by merge items, but for the partition copies,
    // which walk vertex ranges
    if (!part) ASC_TRY(ensure_items(g));
    auto args_of = [&](int parity_in, int region) {
        RegionArgs a = region_args(g, parity_in, region, false);
        if (!part) attach_items(ws, a);
        attach_far(g, algo, a);
        return a;
    };
    uint64_t part_bytes = 0;
    uint32_t part_copies = 0;
    int iters = 0;
    double phase_ms[3] = {0, 0, 0};  // static top-down, on-demand top-down, bottom-up
    const uint32_t nwords = V / 32 + 1;
    // SSSP re-expands, and bottom-up steps reach vertices without expanding
    // them, so reached vertices are counted at the end; a top-down BFS expands
    // every reached vertex exactly once: its expansion counts are the reached ones
    const bool count_reached = algo == ASC_SSSP || (algo == ASC_BFS && ws->bu_active);
    // Connected components without an iteration cap of the caller's: the label of
    // the smallest id with out-edges first. Nothing smaller reaches what it
    // reaches, so those labels are final and each of its lists is read once; with
    // every vertex in the first frontier, nearly all lists are read again when the
    // giant component's label arrives (6 M vertices symmetrised, 180 M edges: 2.39
    // ms against 3.61). A label that spreads slowly (a long path) is joined by the
    // rest after kFirstLabelIterations. The timed, counting and comparison runs
    // start from every vertex.
    const bool first_label = all && p.max_iterations <= 0 && g->E &&
                             !(p.flags & (ASC_RUN_PHASE_TIMING | ASC_RUN_FRAGMENT_COUNTS | ASC_RUN_GATHER_COPY |
                                          ASC_RUN_PARTITION_COPY));
    const uint32_t first =
        first_label ? (uint32_t)(std::upper_bound(g->h_ptr, g->h_ptr + V + 1, 0u) - g->h_ptr) - 1 : source;
    bool rest_waits = first_label && !device_loop;  // the other labels have not started
    const bool want = out && !(p.flags & ASC_RUN_NO_OUTPUT);
    bool values_reported = device_loop && want && !(p.flags & ASC_RUN_DEVICE_OUT) && V <= kReportedValues;
    if (values_reported) {  // only what the host can write to; the copy below answers for the rest
        cudaPointerAttributes attr;
        if (cudaPointerGetAttributes(&attr, out) != cudaSuccess) cudaGetLastError();
        else if (attr.type == cudaMemoryTypeDevice) values_reported = false;
    }
    ASC_CUDA(cudaEventRecord(ws->ev[0], s));
    ASC_CUDA(cudaMemsetAsync(ws->ctl, 0, 4 * CTL_WORDS, s));
    if (device_loop) {
        LoopArgs l;
        memset(&l, 0, sizeof(l));
        for (int parity = 0; parity < 2; parity++) {
            FusedArgs &x = parity ? l.x1 : l.x0;
            x.r0 = args_of(parity, 0);
            x.r1 = args_of(parity, 1);
            x.work = x.r0.cnt_out + 4;
        }
        l.ctl = ws->ctl;
        l.report = ws->h_ctl;
        l.nwords = nwords;
        l.src = first;
        l.all = all && !first_label ? 1 : 0;
        l.first_label = first_label ? 1 : 0;
        l.first_cap = kFirstLabelIterations;
        l.polls = t_barrier_polls;
        l.cap = (uint32_t)std::min<int64_t>(cap, 0x7fffffff);
        l.thresh = 1 + ws->tune.delta;
        l.delta = ws->tune.delta;
        l.count_reached = count_reached ? 1 : 0;
        if (near_far(g, algo)) ASC_CUDA(cudaMemsetAsync(ws->ctl + CTL_MINFAR, 0xff, 16, s));
        const TraverseFn fn = pick_traverse(algo, edge_layout(g));
        uint32_t grid;
        ASC_TRY(loop_grid(g, algo, fn, &grid));
        if (values_reported) l.values = ws->h_ctl + CTL_WORDS;
        ws->h_ctl[CTL_TIMEOUT] = 2;  // stays when a barrier ran out of time and nothing is reported
        void *args[] = {&l};
        ASC_CUDA(cudaLaunchCooperativeKernel((const void *)fn, dim3(grid), dim3(kBlock), args, 0, s));
        launches += 1;
    } else {
        for (int i = 0; i < 2; i++) ASC_CUDA(cudaMemsetAsync(ws->bitmap[i], 0, 4 * (V / 32 + 2), s));
        ASC_CUDA(cudaMemsetAsync(ws->visited, 0, 4 * (V / 32 + 2), s));
        const uint32_t ig = fill_grid(ws, V);
        if (algo == ASC_CC) init_values_kernel<kCC><<<ig, kBlock, 0, s>>>(ws->val, V, 0);
        else if (algo == ASC_BFS) init_values_kernel<kBFS><<<ig, kBlock, 0, s>>>(ws->val, V, source);
        else init_values_kernel<kSSSP><<<ig, kBlock, 0, s>>>(ws->val, V, source);
        if (near_far(g, algo)) {
            ASC_CUDA(cudaMemsetAsync(ws->far_bits, 0, 4 * (V / 32 + 2), s));
            ASC_CUDA(cudaStreamSynchronize(s));  // the staging word below is host memory
            ws->h_ctl[CTL_THRESH] = 1 + ws->tune.delta;
            ASC_CUDA(cudaMemcpyAsync(ws->ctl + CTL_THRESH, ws->h_ctl + CTL_THRESH, 4, cudaMemcpyHostToDevice, s));
        }
        // the seeded frontier lands in parity 0 (as the output of a virtual pass from parity 1)
        RegionArgs sa = args_of(1, 0);
        const bool seed_all = all && !first_label;
        seed_bits_kernel<<<seed_all ? fill_grid(ws, nwords) : 1, kBlock, 0, s>>>(sa, first, seed_all ? 1 : 0, nwords);
        build_frontier_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(sa, ws->bitmap[0], nwords);
        launches += 3;
        ASC_CUDA(cudaGetLastError());
    }
    uint32_t cnt[CTL_BLOCK] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (!device_loop) {
        ASC_CUDA(cudaMemcpyAsync(ws->h_ctl, ws->ctl, 4 * CTL_BLOCK, cudaMemcpyDeviceToHost, s));
        ASC_CUDA(cudaStreamSynchronize(s));
        memcpy(cnt, ws->h_ctl, sizeof(cnt));
    }
    int parity = 0;
    const uint32_t div = ws->tune.dense_div;
    auto region_work = [&](int region) -> uint64_t {
        const uint32_t range = region == 0 ? g->static_vertices : V - g->static_vertices;
        const bool bitmap_mode = div && cnt[6 + region] > range / div;
        if (bitmap_mode && !part && (region || (uint64_t)cnt[6 + region] * ws->item_div > range))
            return region == 0 ? ws->n_items_static : ws->n_items - ws->n_items_static;
        const uint32_t per = bitmap_mode ? (uint32_t)kBlock : kMinTile;
        return (uint64_t)cnt[2 + region] + ((bitmap_mode ? range : cnt[region]) + per - 1) / per;
    };
    while ((cnt[6] | cnt[7]) || rest_waits) {
        if (rest_waits && rest_joins((uint32_t)iters, (uint64_t)cnt[6] + cnt[7], kFirstLabelIterations)) {
            rest_waits = false;
            RegionArgs a = args_of(1 - parity, 0);  // writes this parity's lists
            ASC_CUDA(cudaMemsetAsync(a.cnt_out, 0, 4 * CTL_BLOCK, s));
            seed_unlabelled_kernel<<<fill_grid(ws, V), kBlock, 0, s>>>(a, a.bitmap, first, a.cnt_out + 6);
            build_frontier_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(a, a.bitmap, nwords);
            launches += 2;
            ASC_CUDA(cudaGetLastError());
            ASC_CUDA(cudaMemcpyAsync(ws->h_ctl, a.cnt_out, 4 * CTL_BLOCK, cudaMemcpyDeviceToHost, s));
            ASC_CUDA(cudaStreamSynchronize(s));
            memcpy(cnt, ws->h_ctl, sizeof(cnt));
            continue;
        }
        if (iters >= cap) return fail(ASC_ERR_TIMEOUT, "no fixpoint after %d iterations", iters);
        iters++;
        const int po = 1 - parity;
        ASC_CUDA(cudaMemsetAsync(ws->ctl + CTL_BLOCK * po, 0, 4 * CTL_BLOCK, s));
        ASC_CUDA(cudaMemsetAsync(ws->bitmap[po], 0, 4 * (V / 32 + 2), s));
        if (near_far(g, algo)) ASC_CUDA(cudaMemsetAsync(ws->ctl + CTL_MINFAR, 0xff, 4, s));
        if (gather) {
            // the on-demand list and segments go to the host first, so the host
            // gathers while the static region expands on the device
            ASC_CUDA(cudaMemcpyAsync(ws->h_list, ws->queue[parity] + g->static_vertices, 4ull * cnt[1],
                                     cudaMemcpyDeviceToHost, s));
            ASC_CUDA(cudaMemcpyAsync(ws->h_segs, ws->segs[parity] + ws->segcap_static, 8ull * cnt[3],
                                     cudaMemcpyDeviceToHost, s));
            ASC_CUDA(cudaEventRecord(ws->ev[3], s));
            const uint64_t items0 = region_work(0);
            if (items0) {
                RegionArgs a = args_of(parity, 0);
                expand(g, a, grid_for(ws, items0));
                launches++;
            }
            ASC_TRY(gather_ondemand(g, algo, parity, cnt, ws->ev[3], launches));
        } else if (part) {
            // the static region in place, then every on-demand partition that
            // holds a frontier vertex: copied whole, its frontier expanded from
            // the copy (partition j of this run into buffer j % 2)
            const uint64_t items0 = region_work(0);
            if (items0) {
                RegionArgs a = args_of(parity, 0);
                expand(g, a, grid_for(ws, items0));
                launches++;
            }
            PartPlan *pp = ws->part;
            const uint32_t np = (uint32_t)pp->parts.size();
            if (cnt[7]) {
                part_active_kernel<<<std::min<uint32_t>(np, ws->num_sms * 8), kBlock, 0, s>>>(
                    ws->bitmap[parity], pp->d_ranges, np, pp->d_flags);
                ASC_CUDA(cudaMemsetAsync(pp->d_work, 0, 4ull * np, s));
                ASC_CUDA(cudaMemcpyAsync(pp->h_flags, pp->d_flags, 4ull * np, cudaMemcpyDeviceToHost, s));
                ASC_CUDA(cudaStreamSynchronize(s));
                launches++;
            }
            for (uint32_t k = 0; cnt[7] && k < np; k++) {
                if (!pp->h_flags[k]) continue;
                const Partition &x = pp->parts[k];
                const int b = part_copies & 1;
                ASC_CUDA(cudaStreamWaitEvent(pp->copy, pp->consumed[b], 0));
                ASC_CUDA(cudaMemcpyAsync(g->d_stage[b], g->h_edges + x.w_lo, 4 * x.w_n, cudaMemcpyHostToDevice,
                                         pp->copy));
                ASC_CUDA(cudaEventRecord(pp->copied[b], pp->copy));
                ASC_CUDA(cudaStreamWaitEvent(s, pp->copied[b], 0));
                RegionArgs a = args_of(parity, 1);
                a.edges = (const uint32_t *)((uintptr_t)g->d_stage[b] - 4 * (uintptr_t)x.w_lo);
                a.dense_begin = x.v_lo;
                a.dense_end = x.v_hi;
                a.cnt_in = pp->d_cnt + 8ull * k;  // id-order walk of the range, no segments
                a.dense_div = 0xffffffffu;
                a.huge = 0xffffffffu;             // long lists too are expanded from the copy
                a.work = pp->d_work + k;
                expand(g, a, grid_for(ws, (x.v_hi - (x.v_lo & ~31u) + kBlock - 1) / kBlock));
                ASC_CUDA(cudaEventRecord(pp->consumed[b], s));
                launches++;
                part_copies++;
                part_bytes += 4 * x.w_n;
            }
        } else if (pt.on && ws->bu_active && ws->in_ptr && ((uint64_t)cnt[6] + cnt[7]) * ws->tune.bu_div > V) {
            // diagnostic: a bottom-up step, timed on its own
            RegionArgs a = args_of(parity, 0);
            ASC_TRY(pt.begin(2));
            pt.record(s);
            bottom_up_kernel<<<bu_grid(ws, nwords), kBlock, 0, s>>>(a, nwords, iters + 1);
            pt.record(s);
            launches++;
        } else if (pt.on) {
            // diagnostic: one launch per region, each timed on its own
            for (int region = 0; region < 2; region++) {
                const uint64_t items = region_work(region);
                if (!items) continue;
                RegionArgs a = args_of(parity, region);
                ASC_TRY(pt.begin(region));
                pt.record(s);
                expand(g, a, grid_for(ws, items));
                pt.record(s);
                launches++;
            }
        } else {
            const uint64_t items = region_work(0) + region_work(1);
            FusedArgs x;
            x.r0 = args_of(parity, 0);
            x.r1 = args_of(parity, 1);
            x.work = x.r0.cnt_out + 4;
            fused(s, x, grid_for(ws, items));
            launches++;
            if (algo == ASC_BFS && x.r0.in_ptr) {
                bottom_up_kernel<<<bu_grid(ws, nwords), kBlock, 0, s>>>(x.r0, nwords, iters + 1);
                launches++;
            }
        }
        {
            RegionArgs out_args = args_of(parity, 0);
            if (near_far(g, algo)) {
                launch_far(g, s, out_args);
                launches += 2;
            }
            build_frontier_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(out_args, ws->bitmap[po], nwords);
        }
        launches++;
        ASC_CUDA(cudaGetLastError());
        ASC_CUDA(cudaMemcpyAsync(ws->h_ctl, ws->ctl + CTL_BLOCK * po, 4 * CTL_BLOCK, cudaMemcpyDeviceToHost, s));
        ASC_CUDA(cudaStreamSynchronize(s));
        memcpy(cnt, ws->h_ctl, sizeof(cnt));
        if (pt.on) ASC_TRY(pt.sum(phase_ms));
        parity = po;
        iteration_boundary();
    }
    if (count_reached && !device_loop) {
        if (algo == ASC_BFS)
            reached_bits_kernel<<<fill_grid(ws, 32ull * nwords), kBlock, 0, s>>>(
                ws->visited, g->d_ptr, V, nwords, (unsigned long long *)(ws->ctl + CTL_STATS) + 4);
        else
            reached_kernel<<<fill_grid(ws, V), kBlock, 0, s>>>(ws->val, g->d_ptr, V,
                                                               (unsigned long long *)(ws->ctl + CTL_STATS) + 4);
        launches++;
    }
    ASC_CUDA(cudaEventRecord(ws->ev[1], s));
    ASC_CUDA(cudaGetLastError());
    const bool copies = want && !values_reported;
    if (copies) {
        ASC_CUDA(cudaMemcpyAsync(out, ws->val, 4ull * V,
                                 (p.flags & ASC_RUN_DEVICE_OUT) ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                 s));
        ASC_CUDA(cudaEventRecord(ws->ev[2], s));
    }
    if (!device_loop) ASC_CUDA(cudaMemcpyAsync(ws->h_ctl, ws->ctl, 4 * CTL_WORDS, cudaMemcpyDeviceToHost, s));
    ASC_CUDA(cudaStreamSynchronize(s));
    if (device_loop) {
        if (ws->h_ctl[CTL_TIMEOUT] == 2) return fail(ASC_ERR_TIMEOUT, "a grid barrier ran out of time");
        iters = (int)ws->h_ctl[CTL_ITERS];
        if (ws->h_ctl[CTL_TIMEOUT]) return fail(ASC_ERR_TIMEOUT, "no fixpoint after %d iterations", iters);
        if (values_reported) memcpy(out, ws->h_ctl + CTL_WORDS, 4ull * V);
    }
    if (st) {
        memset(st, 0, sizeof(*st));
        const unsigned long long *hs = (const unsigned long long *)(ws->h_ctl + CTL_STATS);
        const unsigned long long bu_edges = *(const unsigned long long *)(ws->h_ctl + CTL_BU_EDGES);
        st->iterations = iters;
        st->edges_processed = hs[0] + hs[1];
        st->ondemand_edges = hs[1];
        // out-edges in their stored width, in-edges of bottom-up steps in theirs
        const unsigned long long bu_od = ws->in_edges ? 0 : bu_edges;
        st->ondemand_bytes = edge_store_bytes(g, hs[1] - bu_od) + (bu_od * g->in_ebits + 7) / 8;
        if (part) {  // what the partition copies moved
            st->ondemand_bytes = part_bytes;
            st->staged_chunks = part_copies;
        }
        st->bottom_up_edges = bu_edges;
        st->bottom_up_vertices = *(const unsigned long long *)(ws->h_ctl + CTL_BU_VERTS);
        st->frontier_vertices = hs[2] + hs[3];
        st->ondemand_vertices = hs[3];
        if (algo == ASC_CC) {
            st->reached_vertices = V;
            st->reached_edges = g->E;
        } else if (algo == ASC_BFS && !count_reached) {
            st->reached_vertices = hs[2] + hs[3];
            st->reached_edges = hs[0] + hs[1];
        } else {
            st->reached_vertices = hs[4];
            st->reached_edges = hs[5];
        }
        float ms = 0;
        ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[0], ws->ev[1]));
        st->ms_total = ms;
        if (copies) {
            ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[1], ws->ev[2]));
            st->ms_copyout = ms;
        }
        st->ms_static = phase_ms[0];
        st->ms_ondemand = phase_ms[1];
        st->ms_bottom_up = phase_ms[2];
        st->kernel_launches = launches;
    }
    return ASC_OK;
}

// Copies the FP64 ranks out as T: directly for FP64; for FP32 rounded to
// float on the device, into the caller's buffer (ASC_RUN_DEVICE_OUT) or into
// staging (a contribution array, free once the passes are over) copied out.
template <typename T>
asc_status copy_ranks_out(asc_graph *g, const double *rank, void *staging, void *out, uint32_t flags) {
    const uint32_t V = (uint32_t)g->V;
    cudaStream_t s = g->stream;
    const cudaMemcpyKind kind = (flags & ASC_RUN_DEVICE_OUT) ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    if (sizeof(T) == 8) {
        ASC_CUDA(cudaMemcpyAsync(out, rank, 8 * (size_t)V, kind, s));
        return ASC_OK;
    }
    float *dst = (flags & ASC_RUN_DEVICE_OUT) ? (float *)out : (float *)staging;
    pr_rank_to_float_kernel<<<fill_grid(g->ws, V), kBlock, 0, s>>>(rank, dst, V);
    ASC_CUDA(cudaGetLastError());
    if (!(flags & ASC_RUN_DEVICE_OUT)) ASC_CUDA(cudaMemcpyAsync(out, staging, 4 * (size_t)V, kind, s));
    return ASC_OK;
}

template <typename T, bool REF>
static asc_status pagerank_impl(asc_graph *g, const asc_params &p, void *out, asc_stats *st) {
    Workspace *ws = g->ws;
    ASC_TRY(ensure_pr_buffers(g, sizeof(T)));
    const uint32_t V = (uint32_t)g->V;
    cudaStream_t s = g->stream;
    uint32_t launches = 0;
    PhaseTimer pt(ws, (p.flags & ASC_RUN_PHASE_TIMING) != 0);
    typedef typename PrAcc<T>::type Acc;
    double *rank = (double *)ws->pr_rank;
    T *c[2] = {(T *)ws->pr_contrib[0], (T *)ws->pr_contrib[1]};

    ASC_CUDA(cudaEventRecord(ws->ev[0], s));
    ASC_CUDA(cudaMemsetAsync(ws->ctl, 0, 4 * CTL_WORDS, s));
    // the start vector's dangling mass goes to the pair before pass 0's
    pr_init_kernel<T><<<fill_grid(ws, V), kBlock, 0, s>>>(rank, c[0], c[1], (Acc *)ws->pr_sum, g->d_outdeg, V,
                                                          (double *)(ws->ctl + CTL_ACC) + 4);
    launches++;
    RegionArgs sa = base_args(g, 1);  // seeds land in parity 0
    const uint32_t nwords = V / 32 + 1;
    if (REF) {
        // every vertex starts active: full bitmap, then lists/segments from it
        for (int i = 0; i < 2; i++) ASC_CUDA(cudaMemsetAsync(ws->bitmap[i], 0, 4 * (V / 32 + 2), s));
        seed_bits_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(sa, 0, 1, nwords);
        launches++;
    }
    ASC_CUDA(cudaGetLastError());
    // reference mode: this pass's active vertices per region and their in-edges
    uint32_t active[2] = {g->static_vertices, V - g->static_vertices};
    uint64_t active_edges = g->E;
    unsigned long long item_counts[4] = {0, 0, 0, 0};  // of the passes over items

    // standard PageRank on a graph with staging buffers: the on-demand edges are
    // copied in chunks every pass, overlapped with the kernels
    bool staged = false;
    if (!REF && !pt.on && !(p.flags & ASC_RUN_NO_STAGING)) ASC_TRY(ensure_stage_plan(g, &staged));
    StagePlan *sp = staged ? ws->stage : nullptr;
    ASC_TRY(ensure_items(g));

    // REF: the active set alternates parity like a traversal frontier.
    ASC_TRY(ensure_pass_events(ws));
    const int depth = pt.on || staged || t_iteration_hook.fn ? 1 : 2;
    int it = 0, launched = 0;  // passes that ended, that were launched
    bool over_items[kPassSlots] = {};  // a pass in flight runs over items, not lists
    const int max_it = p.max_iterations > 0 ? p.max_iterations : (REF ? 1000000 : 100);
    double residual = 0;
    double phase_ms[2] = {0, 0};
    bool over = false;
    auto wait_pass = [&]() -> asc_status {  // for the oldest pass in flight
        ASC_CUDA(cudaEventSynchronize(ws->pass_ev[it % kPassSlots]));
        if (over_items[it % kPassSlots]) {
            unsigned long long n[4];
            pr_pass_counts(g, 1, n);
            item_counts[0] += n[0];
            item_counts[1] += n[1];
            item_counts[2] += REF ? active[0] : n[2];
            item_counts[3] += REF ? active[1] : n[3];
        }
        const unsigned long long *r = pass_slot(ws, it);
        if (REF) {
            active[0] = (uint32_t)r[0];
            active[1] = (uint32_t)(r[0] >> 32);
            active_edges = r[1];
            over = !(active[0] | active[1]);
        } else {
            memcpy(&residual, r, 8);
            over = residual < p.tolerance;
        }
        if (pt.on) ASC_TRY(pt.sum(phase_ms));
        it++;
        iteration_boundary();
        return ASC_OK;
    };
    for (;;) {
        if (launched - it >= depth || (launched > it && launched >= max_it)) ASC_TRY(wait_pass());
        if (over) break;  // a pass launched after the last one changes nothing
        if (launched >= max_it) {
            if (launched > it) continue;
            if (REF) return fail(ASC_ERR_TIMEOUT, "reference PageRank still active after %d passes", it);
            break;
        }
        // reference mode: lists are made from this pass's own counts; items serve
        // any, so their rule may look at those of the pass before
        if (REF && active_edges <= g->E / kPrDenseDiv && launched > it) {
            ASC_TRY(wait_pass());
            if (over) break;
        }
        const int cp = launched & 1;
        const int parity = cp, po = 1 - cp;
        if (REF) ASC_CUDA(cudaMemsetAsync(ws->bitmap[po], 0, 4 * (V / 32 + 2), s));
        over_items[launched % kPassSlots] = !REF || active_edges > g->E / kPrDenseDiv;
        if (over_items[launched % kPassSlots]) {
            // every row
            PrItemArgs<T> ia;
            memset(&ia, 0, sizeof(ia));
            ia.items = ws->items;
            ia.ptr = g->d_ptr;
            ia.outdeg = g->d_outdeg;
            ia.rank = rank;
            ia.c_old = c[cp];
            ia.c_new = c[1 - cp];
            ia.sum = (Acc *)ws->pr_sum;
            set_pass(ws, p, launched, ia);
            ia.work = ws->ctl + CTL_BLOCK * po + 4;
            ia.V = V;
            ia.ebits = g->ebits;
            ia.bitmap_in = ws->bitmap[parity];
            ia.bitmap = ws->bitmap[po];
            ia.cnt_in = ws->ctl + CTL_BLOCK * parity;
            ia.cnt_out = ws->ctl + CTL_BLOCK * po;
            ia.active_edges = (unsigned long long *)(ws->ctl + CTL_ACTIVE);
            ia.S = g->static_vertices;
            if (staged) ASC_CUDA(cudaMemsetAsync(sp->d_work, 0, 4 * sp->launches.size(), s));
            // one launch for both regions; one per chunk when staged; timed runs
            // launch the regions apart
            const uint32_t runs = staged ? (uint32_t)sp->launches.size() : pt.on ? 2 : 1;
            for (uint32_t k = 0; k < runs; k++) {
                if (staged) {
                    ASC_TRY(stage_chunk(g, sp, k, s, ia.sl));
                    ia.work = sp->d_work + k;
                } else {
                    for (uint32_t r = 0; r < 2; r++) {
                        ia.sl[r] = pr_slice(g, (int)r);
                        if (pt.on && r != k) ia.sl[r].n = 0;
                    }
                }
                const uint32_t n = ia.sl[0].n + ia.sl[1].n;
                if (!n) continue;
                if (pt.on && !staged) ASC_CUDA(cudaMemsetAsync(ia.work, 0, 4, s));
                ASC_TRY(pt.begin((int)k));
                pt.record(s);
                pr_pull_items_kernel<T, REF><<<item_grid(ws, n), kBlock, 0, s>>>(ia);
                pt.record(s);
                if (staged) ASC_TRY(stage_release(sp, k, s));
                launches++;
            }
            pr_cut_rows_kernel<T, REF><<<fill_grid(ws, ws->n_items), kBlock, 0, s>>>(ia, ws->n_items);
            launches++;
        } else {
            // the active vertices' lists and segments, then one launch for both
            // regions (timed runs launch them apart)
            RegionArgs lists = region_args(g, po, 0, false);  // writes the lists of this parity
            build_frontier_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(lists, ws->bitmap[parity], nwords);
            launches++;
            PrArgs pr[2];
            for (int r = 0; r < 2; r++) {
                pr[r].r = region_args(g, parity, r, false);
                pr[r].outdeg = g->d_outdeg;
                pr[r].rank = rank;
                pr[r].c_old = (const double *)c[cp];
                pr[r].c_new = (double *)c[1 - cp];
                pr[r].sum = (double *)ws->pr_sum;
            }
            for (uint32_t k = 0; k < (pt.on ? 2u : 1u); k++) {
                if (pt.on && !active[k]) continue;
                ASC_TRY(pt.begin((int)k));
                pt.record(s);
                pr_pull_lists_kernel<<<(uint32_t)(ws->num_sms * ws->tune.ctas_per_sm), kBlock, 0, s>>>(
                    pr[0], pr[1], pt.on ? 1u << k : 3u);
                pt.record(s);
                launches++;
            }
            const uint64_t segs = ws->segcap_static + ws->segcap_ondemand;
            if (segs) {
                pr_apply_segmented_kernel<<<fill_grid(ws, segs), kBlock, 0, s>>>(
                    pr[0], ws->segs[parity], ws->segs[parity] + ws->segcap_static);
                launches++;
            }
            PrItemArgs<T> ia;
            memset(&ia, 0, sizeof(ia));
            set_pass(ws, p, launched, ia);
            ia.cnt_in = ws->ctl + CTL_BLOCK * parity;
            ia.cnt_out = ws->ctl + CTL_BLOCK * po;
            ia.active_edges = (unsigned long long *)(ws->ctl + CTL_ACTIVE);
            pr_end_pass_kernel<T><<<1, 32, 0, s>>>(ia);
            launches++;
        }
        ASC_CUDA(cudaGetLastError());
        ASC_CUDA(cudaEventRecord(ws->pass_ev[launched % kPassSlots], s));
        launched++;
    }
    ASC_CUDA(cudaEventRecord(ws->ev[1], s));
    if (out && !(p.flags & ASC_RUN_NO_OUTPUT)) {
        ASC_TRY(copy_ranks_out<T>(g, rank, (void *)c[0], out, p.flags));
        launches += sizeof(T) == 4;
    }
    ASC_CUDA(cudaEventRecord(ws->ev[2], s));
    ASC_CUDA(cudaMemcpyAsync(ws->h_ctl + CTL_STATS, ws->ctl + CTL_STATS, 8 * 6, cudaMemcpyDeviceToHost, s));
    ASC_CUDA(cudaStreamSynchronize(s));
    if (st) {
        memset(st, 0, sizeof(*st));
        const unsigned long long *hs = (const unsigned long long *)(ws->h_ctl + CTL_STATS);
        unsigned long long n[4] = {hs[0], hs[1], hs[2], hs[3]};
        for (int k = 0; k < 4; k++) n[k] += item_counts[k];
        st->iterations = it;
        st->edges_processed = n[0] + n[1];
        st->ondemand_edges = n[1];
        st->ondemand_bytes = staged ? sp->copy_bytes * (uint64_t)it : edge_store_bytes(g, n[1]);
        st->staged_chunks = staged ? (uint32_t)(sp->launches.size() * it) : 0;
        st->frontier_vertices = n[2] + n[3];
        st->ondemand_vertices = n[3];
        st->reached_vertices = V;
        st->reached_edges = g->E;
        st->residual = residual;
        float ms = 0;
        ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[0], ws->ev[1]));
        st->ms_total = ms;
        ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[1], ws->ev[2]));
        st->ms_copyout = ms;
        st->ms_static = phase_ms[0];
        st->ms_ondemand = phase_ms[1];
        st->kernel_launches = launches;
    }
    return ASC_OK;
}

// -------------------------------------------- multi-source batches (<= 64) --
//
// Up to 64 BFS or SSSP sources of one graph advance together: each vertex
// carries a 64-bit mask of the sources for which it is in the frontier, so one
// read of an edge serves every source of the batch. BFS keeps 64-bit visited /
// frontier / next masks per vertex and is level-synchronous, so each source's
// levels equal a single-source BFS from it. Batched SSSP keeps a vertex-major
// [V][64] distance block (one 256-byte row per vertex) and relaxes the sources
// of a frontier vertex's mask lane by lane; its fixpoint per source is the
// single-source one. Expansion only ORs masks and marks touched vertices in a
// bitmap; an apply pass over the touched words turns them into the next
// frontier bitmap, and the compaction kernel of the single-query engine builds
// the lists and segments.
//
// Batches are continuous: source slots are filled and emptied between
// iterations. A query joins as soon as a slot (and, for BFS, a level plane) is
// free, advances with the other sources, and leaves when its own frontier is
// empty; levels are counted from the iteration the source joined, so every
// query's values equal a solo run. asc_run_batch is one fill of the slots.
struct BatchEngine {
    asc_graph *g = nullptr;
    bool sssp = false;
    uint32_t stride = 64;             // SSSP distance row length (sources per row)
    Workspace ws;                     // own frontier lists, bitmaps, counters
    unsigned long long *front = nullptr;
    ulonglong2 *masks = nullptr;      // BFS, per vertex: visited and next masks, one 16-byte load
    unsigned long long *next = nullptr;  // SSSP, per vertex: the next mask
    uint32_t *touched = nullptr;      // bitmap of vertices whose next mask went non-zero
    uint32_t *dist = nullptr;         // SSSP [V][stride]
    uint32_t *plane[64] = {nullptr};  // BFS per-slot level planes [V]
    uint32_t **d_plane = nullptr;     // device copy of plane[]
    int32_t *d_lvl_off = nullptr;     // per-slot level offset (level = iteration + offset)
    int32_t lvl_off[64] = {0};
    uint32_t *staging = nullptr;      // SSSP column gather [V]
    // asc_run_batch copies finished rows out while later iterations run: two
    // streams, each with 8 gathered SSSP columns (null: memory was short), made
    // before the first iteration
    cudaStream_t out_stream[2] = {nullptr, nullptr};
    uint32_t *out_rows[2] = {nullptr, nullptr};
    cudaEvent_t out_ready = nullptr;  // the iteration that finished the rows
    cudaStream_t stream = nullptr;
    int parity = 0;
    uint32_t it = 0;                  // iterations run so far
    uint64_t active = 0;              // slots in use
    uint64_t device_bytes = 0;        // beside ws
    uint32_t pend_n = 0, pend_slot[64], pend_src[64];
};

namespace {

enum { CTL_ALIVE = 34 };  // u64 (words 34-35): OR of the new frontier masks of an iteration

struct MsArgs {
    RegionArgs r0, r1;            // frontier lists/segments/bitmaps of both regions (val unused)
    unsigned long long *front;    // sources for which v is in the current frontier
    ulonglong2 *masks;            // BFS, per vertex: x sources that reached it, y those that reached it
                                  // in this iteration (atomicOr)
    unsigned long long *next;     // SSSP: the latter alone (8 bytes per vertex)
    uint32_t *touched;            // bitmap: v's next mask went non-zero this iteration
    uint32_t *work;
    uint32_t *dist;               // SSSP: [V][64]
    uint32_t V;
};

struct MsSmem {
    uint32_t pref[kBlock + 1];
    uint32_t start[kBlock];
    unsigned long long f[kBlock];
    uint32_t warp[kWarps + 1];
    uint32_t work;
};

// BFS relaxation of one edge for a whole mask f; now is the earlier load of v's
// masks. The atomics are fire-and-forget: a thread that saw an empty next mask
// marks v as touched (two may), one that saw it set leaves that to whoever set it,
// and sources already there cost nothing.
__device__ __forceinline__ void ms_reach(const MsArgs &m, uint32_t v, unsigned long long f, ulonglong2 now) {
    const unsigned long long nb = f & ~(now.x | now.y);
    if (!nb) return;
    atomicOr(&m.masks[v].y, nb);
    if (!now.y) atomicOr(&m.touched[v >> 5], 1u << (v & 31));
}

#ifndef ASC_MS_UNROLL
#define ASC_MS_UNROLL 4
#endif
// Edges per thread per pass in the batched BFS expansion (all loads first).
// Regions walked in id order go by merge items with visited and next masks in one
// 16-byte load and atomics only for sources not yet there: 64 sources on RMAT
// scale 21, 3.52 -> 2.4 ms (tiles of 256 vertices and an atomic with a returned
// value per edge and new source before).
// With tiles alone, 8 CTAs per SM: 64-source batch, RMAT scale 22 / 24, 5.45 / 18.27
// ms at 4 edges, 5.58 / 18.46 at 6, 5.78 / 18.96 at 8.
constexpr int kMsUnroll = ASC_MS_UNROLL;
// CTAs per SM (40 registers at 6): 64 sources on RMAT scale 21, 5.33 / 5.28 / 5.51 ms
// at 5 / 6 / 7, the copy of the rows included.
#ifndef ASC_MS_BFS_BLOCKS
#define ASC_MS_BFS_BLOCKS 6
#endif

template <int WORDS>
__device__ void ms_vertices(const MsArgs &m, const RegionArgs &a, bool act, uint32_t u, MsSmem &sm) {
    uint32_t deg = 0, start = 0;
    unsigned long long f = 0;
    if (act && ASC_BAD(u >= m.V, 4, u)) act = false;
    if (act) {
        start = a.ptr[u];
        deg = a.ptr[u + 1] - start;
        if (deg > a.huge) {
            deg = 0;
            act = false;
        }
        f = m.front[u];
    }
    uint32_t total;
    uint32_t excl = block_excl_scan(deg, total, sm.warp);
    sm.pref[threadIdx.x] = excl;
    sm.start[threadIdx.x] = start;
    sm.f[threadIdx.x] = f;
    if (threadIdx.x == 0) sm.pref[kBlock] = total;
    const uint32_t nact = __syncthreads_count(act);
    for (uint32_t base = 0; base < total; base += kMsUnroll * kBlock) {
        uint32_t v[kMsUnroll];
        unsigned long long fk[kMsUnroll];
        ulonglong2 now[kMsUnroll];
#pragma unroll
        for (int k = 0; k < kMsUnroll; k++) {
            const uint32_t e = base + k * kBlock + threadIdx.x;
            v[k] = 0;
            fk[k] = 0;
            if (e < total) {
                int lo = 0, hi = kBlock;
                while (hi - lo > 1) {
                    int mid = (lo + hi) >> 1;
                    if (sm.pref[mid] <= e) lo = mid;
                    else hi = mid;
                }
                const uint64_t idx = (uint64_t)sm.start[lo] + (e - sm.pref[lo]);
                v[k] = WORDS == 2 ? __ldg(a.edges + 2 * idx) : layout_word<WORDS>(a.edges, idx, a.ebits) >> a.wbits;
                fk[k] = sm.f[lo];
                if (ASC_BAD(v[k] >= m.V, 5, v[k])) {
                    v[k] = 0;
                    fk[k] = 0;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kMsUnroll; k++) now[k] = fk[k] ? m.masks[v[k]] : make_ulonglong2(0, 0);
#pragma unroll
        for (int k = 0; k < kMsUnroll; k++) ms_reach(m, v[k], fk[k], now[k]);
    }
    if (threadIdx.x == 0) {
        atomicAdd(&a.stats[a.region], (unsigned long long)total);
        atomicAdd(&a.stats[2 + a.region], (unsigned long long)nact);
    }
    __syncthreads();
}

template <int WORDS>
__device__ void ms_segment(const MsArgs &m, const RegionArgs &a, uint64_t item) {
    const uint32_t u = (uint32_t)(item >> 32), k0 = (uint32_t)item;
    if (ASC_BAD(u >= m.V, 6, u)) return;
    const uint32_t b0 = a.ptr[u], e0 = a.ptr[u + 1];
    const uint64_t b = (uint64_t)b0 + (uint64_t)k0 * a.seg_len;
    const uint64_t e = min((uint64_t)e0, b + a.seg_len);
    const uint32_t n = (uint32_t)(e - b);
    const unsigned long long f = m.front[u];
    for (uint32_t base = 0; base < n; base += kMsUnroll * kBlock) {
        uint32_t v[kMsUnroll];
        ulonglong2 now[kMsUnroll];
        bool ok[kMsUnroll];
#pragma unroll
        for (int k = 0; k < kMsUnroll; k++) {
            const uint32_t j = base + k * kBlock + threadIdx.x;
            ok[k] = j < n;
            v[k] = ok[k] ? (WORDS == 2 ? __ldg(a.edges + 2 * (b + j)) : layout_word<WORDS>(a.edges, b + j, a.ebits) >> a.wbits)
                         : 0;
            if (ok[k] && ASC_BAD(v[k] >= m.V, 5, v[k])) {
                ok[k] = false;
                v[k] = 0;
            }
        }
#pragma unroll
        for (int k = 0; k < kMsUnroll; k++) now[k] = ok[k] ? m.masks[v[k]] : make_ulonglong2(0, 0);
#pragma unroll
        for (int k = 0; k < kMsUnroll; k++) ms_reach(m, v[k], ok[k] ? f : 0ull, now[k]);
    }
    if (threadIdx.x == 0) {
        atomicAdd(&a.stats[a.region], (unsigned long long)n);
        if (k0 == 0) atomicAdd(&a.stats[2 + a.region], 1ull);
    }
}

// A merge item of a region that is walked in id order.
template <int WORDS>
__device__ void ms_merge_item(const MsArgs &m, const RegionArgs &a, uint32_t it,
                              ItemSmem<WORDS, unsigned long long> &sm, uint32_t *counts) {
    uint32_t ne, bit0;
    unsigned long long *value;
    if (!stage_merge_item(a, it, sm, [&](uint32_t u) { return m.front[u]; }, &counts[a.region], &counts[2 + a.region],
                          ne, bit0, value))
        return;
    const uint32_t eb = WORDS == 2 ? 64 : WORDS == 1 ? 32 : a.ebits;
    const uint32_t mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
    const uint32_t x0 = threadIdx.x * kVt;
    uint32_t act, st;
    unsigned long long f;
    if (merge_item_edges(sm, value, ne, x0, act, st, f)) {
#pragma unroll
        for (int k0 = 0; k0 < kVt; k0 += kMsUnroll) {
            uint32_t v[kMsUnroll];
            unsigned long long fk[kMsUnroll];
            ulonglong2 now[kMsUnroll];
#pragma unroll
            for (int k = 0; k < kMsUnroll; k++) {
                v[k] = 0;
                fk[k] = 0;
                if ((act >> (k0 + k)) & 1u) {
                    if (k0 + k > 0 && ((st >> (k0 + k)) & 1u)) f = value[sm.row_at[x0 + k0 + k]];
                    const uint32_t at = bit0 + (x0 + k0 + k) * eb;
                    v[k] = (WORDS == kBitsLayout ? staged_word(sm.pool, at, mask) : sm.pool[at >> 5]) >> a.wbits;
                    fk[k] = f;
                    if (ASC_BAD(v[k] >= m.V, 5, v[k])) {
                        v[k] = 0;
                        fk[k] = 0;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kMsUnroll; k++) now[k] = fk[k] ? m.masks[v[k]] : make_ulonglong2(0, 0);
#pragma unroll
            for (int k = 0; k < kMsUnroll; k++) ms_reach(m, v[k], fk[k], now[k]);
        }
    }
    __syncthreads();
}

template <int WORDS>
union MsExpandSmem {
    MsSmem tile;
    ItemSmem<WORDS, unsigned long long> item;
};

template <int WORDS>
__device__ __forceinline__ void ms_item(const MsArgs &m, const RegionArgs &a, uint32_t w, uint32_t n_in,
                                        uint32_t nseg, bool bitmap, uint32_t per, MsExpandSmem<WORDS> &sm,
                                        uint32_t *counts) {
    if (w < nseg) {
        ms_segment<WORDS>(m, a, a.seg_in[w]);
    } else if (!per) {
        ms_merge_item<WORDS>(m, a, a.item_begin + w, sm.item, counts);
    } else if (!bitmap) {
        const uint32_t i = (w - nseg) * per + threadIdx.x;
        const bool act = threadIdx.x < per && i < n_in;
        ms_vertices<WORDS>(m, a, act, act ? a.q_in[i] : 0, sm.tile);
    } else {
        const uint32_t u = (a.dense_begin & ~31u) + (w - nseg) * kBlock + threadIdx.x;
        const bool act = (region_word(a, u & ~31u) >> (u & 31)) & 1u;
        if (__syncthreads_or(act)) ms_vertices<WORDS>(m, a, act, u, sm.tile);
    }
}

template <int WORDS>
__global__ void __launch_bounds__(kBlock, ASC_MS_BFS_BLOCKS) ms_bfs_expand_kernel(MsArgs m) {
    __shared__ MsExpandSmem<WORDS> sm;
    __shared__ uint32_t s_work, counts[4];  // edges, vertices of merge items per region
    if (threadIdx.x < 4) counts[threadIdx.x] = 0;
    uint32_t n0, s0, i0, t0, n1, s1, i1, t1;
    bool m0, m1;
    region_items_bits(m.r0, m.r0.cnt_in, n0, s0, i0, m0, t0);
    region_items_bits(m.r1, m.r1.cnt_in, n1, s1, i1, m1, t1);
    const uint32_t mm = min(i0, i1), total = i0 + i1;
    for (;;) {
        if (threadIdx.x == 0) s_work = atomicAdd(m.work, 1u);
        __syncthreads();
        const uint32_t w = s_work;
        __syncthreads();
        if (w >= total) break;
        bool od;
        uint32_t local;
        if (w < 2 * mm) {
            od = (w & 1) == 0;
            local = w >> 1;
        } else {
            od = i1 > i0;
            local = mm + (w - 2 * mm);
        }
        if (od) ms_item<WORDS>(m, m.r1, local, n1, s1, m1, t1, sm, counts);
        else ms_item<WORDS>(m, m.r0, local, n0, s0, m0, t0, sm, counts);
    }
    if (threadIdx.x < 4 && counts[threadIdx.x])
        atomicAdd(&m.r0.stats[threadIdx.x], (unsigned long long)counts[threadIdx.x]);
}

// Batched SSSP expansion: one CTA per work item (a tile of frontier vertices,
// or one segment of a long list); the distances of a vertex are one row of
// dist (64 sources: 256 bytes).
#ifndef ASC_MS_SSSP_SPARSE
#define ASC_MS_SSSP_SPARSE 4
#endif
// An edge whose source vertex is active for at most this many sources is
// relaxed lane-per-edge, one 4-byte load per source and row; up to
// kMsQuadSources lane-per-edge a 16-byte quad of sources at a time; above that
// a group of lanes per edge. 64- and 8-source batches on RMAT scale 24 (16 lanes
// per many-source edge): 4-byte loads up to 8 sources and half-warps above: 75 /
// 30 ms; quads for 5-8: 75 / 26 ms; quads up to 12 or 16: 79-81 / 26 ms; quads
// for all above 4: 150 / 26 ms; 4-byte loads up to 16, 32 or 64 sources: 82,
// 101, 179 ms (64 sources).
constexpr int kMsSparseSources = ASC_MS_SSSP_SPARSE;
// Sources whose values a lane of the few-source path loads before comparing.
constexpr int kMsGroup = kMsSparseSources < 8 ? kMsSparseSources : 8;

#ifndef ASC_MS_SSSP_ROWS
#define ASC_MS_SSSP_ROWS 2
#endif
// Edges a lane group of the many-source path loads the distance rows of before
// it compares any of them, so those row reads are in flight together.
constexpr int kMsRows = ASC_MS_SSSP_ROWS;
#ifndef ASC_MS_SSSP_QUAD_SOURCES
#define ASC_MS_SSSP_QUAD_SOURCES 8
#endif
#ifndef ASC_MS_SSSP_QUADS
#define ASC_MS_SSSP_QUADS 2
#endif
// Edges whose source vertex is active for more than kMsSparseSources and at
// most kMsQuadSources sources are relaxed lane-per-edge a 16-byte quad of
// sources at a time (kMsQuads quads in flight); above that a lane group per edge.
constexpr int kMsQuadSources = ASC_MS_SSSP_QUAD_SOURCES;
constexpr int kMsQuads = ASC_MS_SSSP_QUADS;
#ifndef ASC_MS_SSSP_PER_LANE
#define ASC_MS_SSSP_PER_LANE 8
#endif
// Sources per lane of a many-source edge; the lanes sharing the edge are the
// row width over this (4: one 16-byte load per lane, 16 lanes for a 64-source
// row; 8: two loads, 8 lanes; 16: four loads, 4 lanes). 64-source batch on RMAT
// scale 24: 76 ms at 4 per lane (two edges per group in flight), 69 at 8 (two
// in flight), 71 at 8 (one), 71 at 16 (one).
constexpr int kMsPerLane = ASC_MS_SSSP_PER_LANE;
static_assert(kMsPerLane == 4 || kMsPerLane == 8 || kMsPerLane == 16, "4, 8 or 16 sources per lane");
// Distance rows of a batch hold R = 16, 32 or 64 sources (R x 4 bytes per
// vertex): the 64-wide batch, or a narrower one where a device budget cannot
// hold 64 columns of a large graph.
__host__ __device__ constexpr bool ms_row_ok(int R) { return R == 16 || R == 32 || R == 64; }

struct MsSsspSmem {
    uint32_t pref[kBlock + 1];       // exclusive degree prefix of the tile's vertices
    uint32_t start[kBlock];          // first edge of each
    uint32_t vid[kBlock];            // vertex id of each
    unsigned long long f[kBlock];    // frontier mask of each
    uint32_t warp[kWarps + 1];
    uint32_t work;
    uint32_t dv[kWarps][32];         // per warp: many-source edges of the current chunk
    uint32_t dw[kWarps][32];
    uint32_t downer[kWarps][32];
};

__device__ __forceinline__ void ms_sssp_load_edge(const RegionArgs &a, uint64_t idx, uint32_t &v, uint32_t &w) {
    if (a.wbits) {
        const uint32_t e = edge_word(a.edges, idx, a.ebits);
        v = e >> a.wbits;
        w = e & ((1u << a.wbits) - 1u);
    } else {
        const uint2 e = __ldg(reinterpret_cast<const uint2 *>(a.edges) + idx);
        v = e.x;
        w = e.y;
    }
}

// Lowers *p to nd when cur, loaded earlier, is larger, and then sets bit in imp:
// a compare and two predicated instructions. Fire-and-forget: a value lowered
// further meanwhile is marked all the same, which costs at most one more
// relaxation. Callers need not test which of a row's sources are active at u (715 M
// warp instructions with those tests and a branch per source on 16.8 M edges of 64
// sources, 60% of the issue slots; bound by them): every column is one that no edge
// improves, but for its source's active vertices. A source not active at u has not
// changed there since it relaxed this edge; a finished one is at its fixpoint; a
// column without a source holds V + 1 everywhere (batch_create, batch_clear), and
// V + 1 plus a weight does not wrap (graphs whose weights could are refused).
__device__ __forceinline__ void relax_min(uint32_t *p, uint32_t nd, uint32_t cur, uint32_t &imp, uint32_t bit) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.lt.u32 q, %2, %3;\n\t"
        "@q red.relaxed.gpu.global.min.u32 [%1], %2;\n\t"
        "@q or.b32 %0, %0, %4;\n\t}"
        : "+r"(imp)
        : "l"(p), "r"(nd), "r"(cur), "r"(bit)
        : "memory");
}

// Marks v as reached for the sources in imp: 32-bit halves, as every atomic of
// the batched SSSP on these masks.
__device__ __forceinline__ void ms_sssp_mark(const MsArgs &m, uint32_t v, unsigned long long imp) {
    uint32_t *next = reinterpret_cast<uint32_t *>(m.next + v);
    if ((uint32_t)imp) atomicOr(next, (uint32_t)imp);
    if ((uint32_t)(imp >> 32)) atomicOr(next + 1, (uint32_t)(imp >> 32));
    atomicOr(&m.touched[v >> 5], 1u << (v & 31));
}

// Relaxes one edge (u -> v, weight w) for the sources in f, lane-per-edge:
// the lane reads the two distance rows a 16-byte quad (four sources) at a
// time, only the quads with an active source, kMsQuads quads in flight.
template <int R>
__device__ __forceinline__ void ms_sssp_lane_quads(const MsArgs &m, uint32_t u, uint32_t v, uint32_t w,
                                                   unsigned long long f) {
    const uint4 *urow = reinterpret_cast<const uint4 *>(m.dist + (uint64_t)u * R);
    uint32_t *vrow = m.dist + (uint64_t)v * R;
    uint32_t qm = 0;
#pragma unroll
    for (int q = 0; q < R / 4; q++) qm |= ((f >> (4 * q)) & 0xfull) ? 1u << q : 0u;
    unsigned long long imp = 0;
    while (qm) {
        int qx[kMsQuads];
        uint4 du[kMsQuads], cur[kMsQuads];
#pragma unroll
        for (int k = 0; k < kMsQuads; k++) {
            qx[k] = qm ? __ffs(qm) - 1 : -1;
            qm &= qm - 1;
            du[k] = make_uint4(0, 0, 0, 0);
            cur[k] = make_uint4(0, 0, 0, 0);
            if (qx[k] >= 0) {
                du[k] = urow[qx[k]];
                cur[k] = reinterpret_cast<const uint4 *>(vrow)[qx[k]];
            }
        }
#pragma unroll
        for (int k = 0; k < kMsQuads; k++) {
            if (qx[k] < 0) continue;
            uint32_t *r = vrow + 4 * qx[k];
            uint32_t bits = 0;
            relax_min(r + 0, du[k].x + w, cur[k].x, bits, 1u);
            relax_min(r + 1, du[k].y + w, cur[k].y, bits, 2u);
            relax_min(r + 2, du[k].z + w, cur[k].z, bits, 4u);
            relax_min(r + 3, du[k].w + w, cur[k].w, bits, 8u);
            imp |= (unsigned long long)bits << (4 * qx[k]);
        }
    }
    if (imp) ms_sssp_mark(m, v, imp);
}

// One warp relaxes 32 consecutive edges of the tile's flattened edge range
// [e0, e0 + 32) ∩ [0, total). An edge whose source vertex is active for at most
// kMsQuadSources sources is relaxed by its own lane for each of them; the
// others are gathered into the warp's shared slots and relaxed by groups of
// R / kMsPerLane lanes, each lane kMsPerLane sources (16-byte loads of the
// source's and the destination's distance rows of R x 4 bytes), kMsRows edges
// per group in flight.
template <int R>
__device__ __forceinline__ void ms_sssp_chunk(const MsArgs &m, const RegionArgs &a, MsSsspSmem &sm, uint32_t e0,
                                              uint32_t total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t e = e0 + lane;
    const bool ok = e < total;
    uint32_t o = 0, v = 0, w = 0;
    unsigned long long f = 0;
    if (ok) {
        int lo = 0, hi = kBlock;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (sm.pref[mid] <= e) lo = mid;
            else hi = mid;
        }
        o = (uint32_t)lo;
        ms_sssp_load_edge(a, (uint64_t)sm.start[o] + (e - sm.pref[o]), v, w);
        f = sm.f[o];
        if (ASC_BAD(v >= m.V || (f >> 1 >> (R - 1)) != 0, 8, v)) {
            v = 0;
            f = 0;
        }
    }
    const int nsrc = __popcll(f);
    const bool dense = nsrc > kMsQuadSources, mid = nsrc > kMsSparseSources && !dense;
    if (ok && nsrc && nsrc <= kMsSparseSources) {
        // few sources: this lane relaxes its edge for each of them, loading the
        // values of kMsGroup sources before comparing any
        const uint32_t u = sm.vid[o];
        uint32_t *row = m.dist + (uint64_t)v * R;
        unsigned long long fm = f, imp = 0;
        while (fm) {
            uint32_t ds[kMsGroup], cur[kMsGroup];
            int sx[kMsGroup];
#pragma unroll
            for (int k = 0; k < kMsGroup; k++) {
                sx[k] = fm ? __ffsll((long long)fm) - 1 : -1;
                fm &= fm - 1;
                ds[k] = sx[k] >= 0 ? m.dist[(uint64_t)u * R + sx[k]] : 0u;
                cur[k] = sx[k] >= 0 ? row[sx[k]] : 0u;
            }
#pragma unroll
            for (int k = 0; k < kMsGroup; k++) {
                const uint32_t nd = ds[k] + w;
                // fire-and-forget lowering: a source lowered further meanwhile
                // (or whose loaded value was stale) is marked active for v all
                // the same, which costs at most one more relaxation and never
                // changes the fixpoint
                if (sx[k] >= 0 && nd < cur[k]) {
                    atomicMin(&row[sx[k]], nd);
                    imp |= 1ull << sx[k];
                }
            }
        }
        if (imp) ms_sssp_mark(m, v, imp);
    }
    if (ok && mid) ms_sssp_lane_quads<R>(m, sm.vid[o], v, w, f);
    const uint32_t dm = __ballot_sync(kFull, ok && dense);
    if (!dm) return;
    if (ok && dense) {
        const uint32_t r = __popc(dm & ((1u << lane) - 1u));
        sm.dv[wid][r] = v;
        sm.dw[wid][r] = w;
        sm.downer[wid][r] = o;
    }
    __syncwarp();
    const uint32_t nd = __popc(dm);
    // R / kMsPerLane lanes per edge, kMsPerLane sources (kMsPerLane / 4 quads) per lane
    constexpr int S = kMsPerLane < R ? kMsPerLane : R, G = R / S, Q = S / 4, EPW = 32 / G;
    const uint32_t grp = (uint32_t)lane / G, l = (uint32_t)lane % G;
    for (uint32_t j0 = 0; j0 < nd; j0 += EPW * kMsRows) {
        uint32_t vk[kMsRows], wk[kMsRows], act[kMsRows];
        uint4 du[kMsRows][Q], cur[kMsRows][Q];
#pragma unroll
        for (int k = 0; k < kMsRows; k++) {
            const uint32_t j = j0 + EPW * k + grp;
            act[k] = 0;
            vk[k] = 0;
            wk[k] = 0;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                du[k][q] = make_uint4(0, 0, 0, 0);
                cur[k][q] = make_uint4(0, 0, 0, 0);
            }
            if (j < nd) {
                const uint32_t ow = sm.downer[wid][j];
                vk[k] = sm.dv[wid][j];
                wk[k] = sm.dw[wid][j];
                act[k] = (uint32_t)(sm.f[ow] >> (S * l)) & (uint32_t)((1ull << S) - 1);
                if (act[k]) {
                    const uint4 *ur = reinterpret_cast<const uint4 *>(m.dist + (uint64_t)sm.vid[ow] * R);
                    const uint4 *vr = reinterpret_cast<const uint4 *>(m.dist + (uint64_t)vk[k] * R);
#pragma unroll
                    for (int q = 0; q < Q; q++) {
                        du[k][q] = ur[Q * l + q];
                        cur[k][q] = vr[Q * l + q];
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kMsRows; k++) {
            const uint32_t j = j0 + EPW * k + grp;
            uint32_t imp = 0;
            if (act[k]) {
                uint32_t *row = m.dist + (uint64_t)vk[k] * R + S * l;
#pragma unroll
                for (int q = 0; q < Q; q++) {
                    relax_min(row + 4 * q + 0, du[k][q].x + wk[k], cur[k][q].x, imp, 1u << (4 * q));
                    relax_min(row + 4 * q + 1, du[k][q].y + wk[k], cur[k][q].y, imp, 2u << (4 * q));
                    relax_min(row + 4 * q + 2, du[k][q].z + wk[k], cur[k][q].z, imp, 4u << (4 * q));
                    relax_min(row + 4 * q + 3, du[k][q].w + wk[k], cur[k][q].w, imp, 8u << (4 * q));
                }
            }
            // the improved sources of the H lanes that share a 32-bit half
            constexpr int H = 32 / S < G ? 32 / S : G;
            uint32_t im = imp << (S * (l % H));
#pragma unroll
            for (int d = H / 2; d > 0; d >>= 1) im |= __shfl_xor_sync(kFull, im, d);
            if (l % H == 0 && j < nd && im) {
                atomicOr(reinterpret_cast<uint32_t *>(m.next + vk[k]) + l / H, im);
                atomicOr(&m.touched[vk[k] >> 5], 1u << (vk[k] & 31));
            }
        }
    }
    __syncwarp();  // the slots are rewritten by the next chunk
}

// One work item of the batched SSSP: a tile of up to 256 list vertices or one
// segment of a long list. The tile's edges are walked as one flattened range,
// 32 per warp per pass, so short lists do not leave lanes idle and every warp
// has loads in flight.
template <int R>
__device__ void ms_sssp_item(const MsArgs &m, const RegionArgs &a, uint32_t w, uint32_t n_in, uint32_t nseg,
                             uint32_t per, MsSsspSmem &sm) {
    bool act = false;
    uint32_t u = 0, start = 0, deg = 0;
    unsigned long long f = 0;
    bool seg = w < nseg;
    if (seg) {
        if (threadIdx.x == 0 && !ASC_BAD((uint32_t)(a.seg_in[w] >> 32) >= m.V, 7, a.seg_in[w] >> 32)) {
            const uint64_t item = a.seg_in[w];
            const uint32_t k0 = (uint32_t)item;
            u = (uint32_t)(item >> 32);
            const uint32_t b0 = a.ptr[u], e0 = a.ptr[u + 1];
            const uint64_t b = (uint64_t)b0 + (uint64_t)k0 * a.seg_len;
            start = (uint32_t)b;
            deg = (uint32_t)(min((uint64_t)e0, b + a.seg_len) - b);
            act = k0 == 0;  // the vertex counts once
            f = m.front[u];
        }
    } else {
        const uint32_t i = (w - nseg) * per + threadIdx.x;
        if (threadIdx.x < per && i < n_in && !ASC_BAD(a.q_in[i] >= m.V, 7, a.q_in[i])) {
            u = a.q_in[i];
            start = a.ptr[u];
            deg = a.ptr[u + 1] - start;
            act = true;
            f = m.front[u];
        }
    }
    uint32_t total;
    const uint32_t excl = block_excl_scan(deg, total, sm.warp);
    sm.pref[threadIdx.x] = excl;
    sm.start[threadIdx.x] = start;
    sm.vid[threadIdx.x] = u;
    sm.f[threadIdx.x] = f;
    if (threadIdx.x == 0) sm.pref[kBlock] = total;
    const uint32_t nact = __syncthreads_count(act);
    for (uint32_t base = 0; base < total; base += kBlock)
        ms_sssp_chunk<R>(m, a, sm, base + (threadIdx.x & ~31u), total);
    if (threadIdx.x == 0) {
        atomicAdd(&a.stats[a.region], (unsigned long long)total);
        atomicAdd(&a.stats[2 + a.region], (unsigned long long)nact);
    }
    __syncthreads();
}

// Work items are per CTA: the static region's segments and list tiles and the
// on-demand region's, interleaved so link-bound and HBM-bound work overlap.
// The SSSP batch always builds lists (its RegionArgs carry dense_div = 0).
template <int R>
__global__ void __launch_bounds__(kBlock, ASC_MS_MIN_BLOCKS) ms_sssp_expand_kernel(MsArgs m) {
    static_assert(ms_row_ok(R), "rows of 16, 32 or 64 sources");
    __shared__ MsSsspSmem sm;
    uint32_t n0, s0, i0, t0, n1, s1, i1, t1;
    bool m0, m1;
    region_items_bits(m.r0, m.r0.cnt_in, n0, s0, i0, m0, t0);
    region_items_bits(m.r1, m.r1.cnt_in, n1, s1, i1, m1, t1);
    const uint32_t mm = min(i0, i1), total = i0 + i1;
    for (;;) {
        if (threadIdx.x == 0) sm.work = atomicAdd(m.work, 1u);
        __syncthreads();
        const uint32_t w = sm.work;
        __syncthreads();
        if (w >= total) break;
        bool od;
        uint32_t local;
        if (w < 2 * mm) {
            od = (w & 1) == 0;
            local = w >> 1;
        } else {
            od = i1 > i0;
            local = mm + (w - 2 * mm);
        }
        if (od) ms_sssp_item<R>(m, m.r1, local, n1, s1, t1, sm);
        else ms_sssp_item<R>(m, m.r0, local, n0, s0, t0, sm);
    }
}

#ifndef ASC_MS_APPLY_WORDS
#define ASC_MS_APPLY_WORDS 4
#endif
constexpr uint32_t kApplyWords = ASC_MS_APPLY_WORDS;

// Apply pass over the touched bitmap: the new sources of a touched vertex
// become its frontier mask, BFS levels are written into the
// sources' planes, and the vertex's bit goes into the next frontier bitmap
// (with per-region counts for the compaction kernel). ORs every new mask into
// *alive so finished sources can be told apart.
template <bool BFS>
__global__ void ms_apply_kernel(MsArgs m, uint32_t **planes, const int32_t *lvl_off, uint32_t it,
                                unsigned long long *alive, uint32_t nwords) {
    // a warp takes kApplyWords touched-bitmap words at a time and walks the non-empty
    // ones, lane = vertex: the level stores of one source go to 32 consecutive
    // entries of its plane (one coalesced store per source present in the word)
    const RegionArgs &a = m.r0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    unsigned long long any = 0;
    uint32_t n0 = 0, n1 = 0;
    for (uint64_t g0 = (uint64_t)warp * kApplyWords; g0 < nwords; g0 += (uint64_t)nwarps * kApplyWords) {
        const uint64_t gw = g0 + lane;
        const uint32_t tw = lane < kApplyWords && gw < nwords ? m.touched[gw] : 0u;
        unsigned nz = __ballot_sync(kFull, tw != 0);
        while (nz) {
            const int j = __ffs(nz) - 1;
            nz &= nz - 1;
            const uint32_t w = (uint32_t)g0 + (uint32_t)j;
            const uint32_t word = __shfl_sync(kFull, tw, j);
            const uint32_t v = 32 * w + lane;
            unsigned long long nb = 0;
            if ((word >> lane) & 1u) {
                if (BFS) {
                    const ulonglong2 now = m.masks[v];
                    nb = now.y & ~now.x;
                    m.masks[v] = make_ulonglong2(now.x | nb, 0);
                } else {
                    nb = m.next[v];
                    m.next[v] = 0;
                }
                m.front[v] = nb;
                any |= nb;
            }
            if (BFS) {
                unsigned long long un = ((unsigned long long)__reduce_or_sync(kFull, (uint32_t)(nb >> 32)) << 32) |
                                        __reduce_or_sync(kFull, (uint32_t)nb);
                while (un) {
                    const int src = __ffsll((long long)un) - 1;
                    un &= un - 1;
                    if (((nb >> src) & 1ull) && !ASC_BAD(!planes[src], 12, src))
                        planes[src][v] = (uint32_t)((int32_t)it + lvl_off[src]);
                }
            }
            const unsigned nbits = __ballot_sync(kFull, nb != 0ull);
            if (lane == 0) {
                m.touched[w] = 0;
                if (nbits) {
                    a.bitmap[w] = nbits;
                    const uint32_t v0 = 32 * w;
                    const uint32_t smask =
                        v0 + 32 <= a.S ? 0xffffffffu : (v0 >= a.S ? 0 : (1u << (a.S - v0)) - 1u);
                    n0 += __popc(nbits & smask);
                    n1 += __popc(nbits & ~smask);
                }
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) any |= __shfl_down_sync(kFull, any, d);
    if (lane == 0) {
        if (any) atomicOr(alive, any);
        if (n0) atomicAdd(&a.cnt_out[6], n0);
        if (n1) atomicAdd(&a.cnt_out[7], n1);
    }
}

struct Admit {
    uint32_t n;
    uint32_t slot[64];
    uint32_t src[64];
};

// Resets the per-slot state of newly admitted slots: BFS clears their bits in
// every visited mask and fills their level planes, SSSP resets their distance
// columns.
__global__ void cb_clear_kernel(ulonglong2 *masks, uint32_t *dist, uint32_t stride, uint32_t **planes,
                                unsigned long long newmask, uint32_t V, uint32_t fill, uint32_t sssp) {
    if (sssp) {
        // stride / 4 lanes per distance row (16 for 64 sources): lane l owns
        // sources 4l..4l+3, one 16-byte store when all four are new, else a merge
        const uint32_t lanes = stride / 4;
        const uint32_t l = threadIdx.x % lanes;
        const uint32_t m4 = (uint32_t)(newmask >> (4 * l)) & 0xfu;
        if (!m4) return;
        const uint64_t h0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / lanes;
        const uint64_t hs = ((uint64_t)gridDim.x * blockDim.x) / lanes;
        for (uint64_t v = h0; v < V; v += hs) {
            uint4 *p = reinterpret_cast<uint4 *>(dist + v * stride) + l;
            uint4 x = make_uint4(fill, fill, fill, fill);
            if (m4 != 0xfu) {
                const uint4 o = *p;
                if (!(m4 & 1u)) x.x = o.x;
                if (!(m4 & 2u)) x.y = o.y;
                if (!(m4 & 4u)) x.z = o.z;
                if (!(m4 & 8u)) x.w = o.w;
            }
            *p = x;
        }
        return;
    }
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        unsigned long long t = newmask;
        masks[v].x &= ~newmask;
        while (t) {
            const int s = __ffsll((long long)t) - 1;
            t &= t - 1;
            if (!ASC_BAD(!planes[s], 11, s)) planes[s][v] = fill;
        }
    }
}

// Admission, phase 1: a new source that is not in the current frontier gets a
// fresh frontier mask (front[] of non-members may hold stale bits).
__global__ void cb_admit_reset_kernel(Admit ad, unsigned long long *front, const uint32_t *bitmap_cur) {
    const uint32_t i = threadIdx.x;
    if (i < ad.n) {
        const uint32_t v = ad.src[i];
        if (!((bitmap_cur[v >> 5] >> (v & 31)) & 1u)) front[v] = 0;
    }
}

// Admission, phase 2: marks each source at level / distance 1 and adds it to
// the current frontier: a vertex that was not a member gets its bit and its
// region count, and joins its region list (or, for a long list, the segment
// list). A region walked through its bitmap ignores the list.
__global__ void cb_admit_kernel(Admit ad, MsArgs m, RegionArgs cur, uint32_t **planes, uint32_t stride,
                                uint32_t sssp) {
    const uint32_t i = threadIdx.x;
    if (i >= ad.n) return;
    const uint32_t s = ad.slot[i], v = ad.src[i];
    if (ASC_BAD(v >= m.V || s >= stride || (!sssp && !planes[s]), 9, v)) return;
    const unsigned long long bit = 1ull << s;
    if (sssp) m.dist[(uint64_t)v * stride + s] = 1;
    else {
        atomicOr(&m.masks[v].x, bit);
        planes[s][v] = 1;
    }
    atomicOr(&m.front[v], bit);
    const uint32_t vb = 1u << (v & 31);
    if (atomicOr(&cur.bitmap[v >> 5], vb) & vb) return;  // already in the frontier
    const bool od = v >= cur.S;
    atomicAdd(&cur.cnt_out[6 + od], 1u);
    const uint32_t deg = cur.ptr[v + 1] - cur.ptr[v];
    if (deg > cur.huge) {
        const uint32_t nseg = (deg + cur.seg_len - 1) / cur.seg_len;
        const uint32_t sb = atomicAdd(&cur.cnt_out[2 + od], nseg);
        if (ASC_BAD((uint64_t)sb + nseg > (od ? cur.segcap_ondemand : cur.segcap_static), 10, sb)) return;
        uint64_t *dst = cur.seg_out + (od ? cur.segcap_static : 0) + sb;
        for (uint32_t k = 0; k < nseg; k++) dst[k] = ((uint64_t)v << 32) | k;
    } else {
        const uint32_t pos = atomicAdd(&cur.cnt_out[od], 1u);
        if (ASC_BAD((od ? cur.S : 0) + pos >= (od ? cur.V : cur.S), 10, pos)) return;
        cur.q_out[(od ? cur.S : 0) + pos] = v;
    }
}

__global__ void cb_gather_column_kernel(const uint32_t *dist, uint32_t stride, uint32_t s, uint32_t *out, uint32_t V) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        out[v] = dist[(uint64_t)v * stride + s];
}

// Columns 8 * group .. + 7 of the distance rows whose bits are set in cols, as
// rows of V values each: a thread reads a vertex's 32 bytes (one sector), and
// each column's stores are consecutive.
__global__ void cb_gather_columns_kernel(const uint32_t *dist, uint32_t stride, uint32_t group, uint32_t cols,
                                         uint32_t *out, uint32_t V) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const uint4 *p = reinterpret_cast<const uint4 *>(dist + (uint64_t)v * stride + 8 * group);
        const uint4 a = p[0], b = p[1];
        const uint32_t x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 8; k++)
            if ((cols >> k) & 1u) out[(uint64_t)k * V + v] = x[k];
    }
}

}  // namespace

uint64_t batch_state_bytes(asc_graph *g, bool sssp, uint32_t stride) {
    const uint64_t V = g->V;
    uint64_t b = (sssp ? 16 : 24) * V + 4 * (V / 32 + 2) + 16 * V + 4 * 4 * (V / 32 + 2) + 8 * (g->E / 256 + 1024) + 4096;
    if (!sssp) b += items_bytes(V, g->E);
    if (sssp) b += 4ull * V * stride + 4 * V;
    return b;
}

uint64_t batch_plane_bytes(asc_graph *g) { return 4ull * g->V; }

thread_local IterationHook t_iteration_hook;

// Self-checking build: the first index check that failed since the last call
// (after the launching stream was synchronized), as an error.
asc_status self_check_result() {
#ifdef ASC_SELF_CHECK
    unsigned long long v = 0;
    ASC_CUDA(cudaMemcpyFromSymbol(&v, g_self_check, sizeof(v)));
    if (v) {
        const unsigned long long zero = 0;
        ASC_CUDA(cudaMemcpyToSymbol(g_self_check, &zero, sizeof(zero)));
        return fail(ASC_ERR_CUDA, "self-check failed at site %u, index %u", (unsigned)(v >> 32), (unsigned)v);
    }
#endif
    return ASC_OK;
}

// Device bytes a graph's single-query state needs (an upper bound before the
// first run; exact afterwards), with the PageRank buffers when asked for.
uint64_t workspace_bytes(asc_graph *g, bool pagerank) {
    const uint64_t V = g->V, E = g->E;
    const Tuning t = g->ws ? g->ws->tune : (g->has_tuning ? g->tuning : Tuning());
    uint64_t b;
    if (g->ws) {
        b = g->ws->device_bytes;
    } else {
        // alloc_workspace: values, two queues, five bitmaps, control words, and
        // two segment lists plus the list of long-list vertices (a list of d >
        // huge_degree edges is ceil(d / segment_edges) <= d / segment_edges + 1
        // segments, and there are at most E / (huge_degree + 1) such lists)
        const uint64_t huge = E / ((uint64_t)t.huge_degree + 1) + 1;
        const uint64_t segs = E / std::max<uint32_t>(1, t.segment_edges) + huge;
        b = 12 * V + 20 * (V / 32 + 2) + 4 * CTL_WORDS + 16 * segs + 4 * huge + 8 * 16;
    }
    if (pagerank && (!g->ws || !g->ws->pr_rank)) b += 4ull * 8 * V;
    if (!g->ws || !g->ws->items) b += items_bytes(V, E);
    if (pagerank && (!g->ws || !g->ws->pr_hot)) b += 8 * kPrHot;
    // in-edge offsets of bottom-up BFS steps, allocated on the first BFS (with
    // the in-edges themselves when every out-edge is resident)
    if (!g->is_csc && t.bu_div && (!g->ws || !g->ws->in_ptr)) {
        b += 4 * (V + 1) + 4 * (V / 32 + 2);
        if (g->static_edges >= E) b += 4 * in_edge_words(g);
    }
    return b;
}

void batch_destroy(BatchEngine *b) {
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    free_ws_buffers(&b->ws);
    for (void *p : {(void *)b->masks, (void *)b->next, (void *)b->front, (void *)b->touched, (void *)b->dist,
                    (void *)b->d_plane, (void *)b->d_lvl_off, (void *)b->staging})
        if (p) cudaFree(p);
    for (auto p : b->plane)
        if (p) cudaFree(p);
    for (int i = 0; i < 2; i++) {
        if (b->out_stream[i]) {
            cudaStreamSynchronize(b->out_stream[i]);
            cudaStreamDestroy(b->out_stream[i]);
        }
        if (b->out_rows[i]) cudaFree(b->out_rows[i]);
    }
    if (b->out_ready) cudaEventDestroy(b->out_ready);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

// Device memory of a batch. Tests make one of a thread's allocations fail as if
// memory had run out: the one after t_allocs_left more (negative: none).
static thread_local int t_allocs_left = -1;
static asc_status batch_alloc(BatchEngine *b, void **p, uint64_t n) {
    cudaError_t e = cudaErrorMemoryAllocation;
    if (t_allocs_left != 0) e = cudaMalloc(p, n ? n : 16);
    if (t_allocs_left >= 0) t_allocs_left--;
    if (e == cudaSuccess) b->device_bytes += n;
    return e == cudaSuccess ? ASC_OK : cuda_fail(e, "cudaMalloc(batch)", __FILE__, __LINE__);
}

extern "C" void asc_test_fail_batch_alloc(int after) { t_allocs_left = after; }
extern "C" void asc_test_barrier_polls(uint32_t polls) { t_barrier_polls = polls; }

// Empties a batch, on its stream: no source, no frontier (lists, bitmaps, counts,
// front masks), no masks. A source dropped without this would leave its frontier to
// whichever source takes its slot next. SSSP: the distance columns of the slots in
// `columns` become those of a source that reaches nothing, since iterations relax
// them along with the columns beside them (see relax_min).
static asc_status batch_clear(BatchEngine *b, uint64_t columns) {
    const uint64_t V = b->g->V;
    b->active = 0;
    b->pend_n = 0;
    ASC_CUDA(cudaMemsetAsync(b->ws.ctl, 0, 4 * CTL_WORDS, b->stream));
    for (auto q : {b->ws.bitmap[0], b->ws.bitmap[1], b->touched})
        ASC_CUDA(cudaMemsetAsync(q, 0, 4 * (V / 32 + 2), b->stream));
    if (b->sssp) ASC_CUDA(cudaMemsetAsync(b->next, 0, 8 * V, b->stream));
    else ASC_CUDA(cudaMemsetAsync(b->masks, 0, 16 * V, b->stream));
    ASC_CUDA(cudaMemsetAsync(b->front, 0, 8 * V, b->stream));
    if (b->sssp && columns) {
        cb_clear_kernel<<<fill_grid(&b->ws, V), kBlock, 0, b->stream>>>(b->masks, b->dist, b->stride, b->d_plane,
                                                                        columns, (uint32_t)V, (uint32_t)V + 1, 1);
        ASC_CUDA(cudaGetLastError());
    }
    return ASC_OK;
}

asc_status batch_create(asc_graph *g, bool sssp, uint32_t stride, BatchEngine **out) {
    BatchEngine *b = new BatchEngine();
    b->g = g;
    b->sssp = sssp;
    b->stride = stride;
    asc_status st = stride == 64 || (sssp && (stride == 16 || stride == 32))
                        ? ASC_OK
                        : fail(ASC_ERR_UNSUPPORTED, "batch rows of %u sources", stride);
    // 64-source batches keep the default thresholds: a graph's tuning is chosen on
    // single-source runs, and the batch kernels measured faster with the defaults
    if (st == ASC_OK) st = alloc_workspace(g, &b->ws, false);
    if (sssp) b->ws.tune.dense_div = 0;  // the SSSP batch walks lists only
    const uint64_t V = g->V;
    auto al = [&](void **p, size_t n) {
        if (st == ASC_OK) st = batch_alloc(b, p, n);
    };
    if (sssp) al((void **)&b->next, 8 * V);
    else al((void **)&b->masks, 16 * V);
    al((void **)&b->front, 8 * V);
    al((void **)&b->touched, 4 * (V / 32 + 2));
    al((void **)&b->d_plane, 8 * 64);
    al((void **)&b->d_lvl_off, 4 * 64);
    if (sssp) {
        al((void **)&b->dist, 4ull * V * stride);
        al((void **)&b->staging, 4 * V);
    }
    if (st == ASC_OK) {
        cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) st = cuda_fail(e, "cudaStreamCreate", __FILE__, __LINE__);
    }
    if (st == ASC_OK && !sssp) st = ensure_items(g, &b->ws, b->stream);
    if (st == ASC_OK) st = batch_clear(b, ~0ull);
    if (st == ASC_OK) {
        cudaError_t e = cudaMemsetAsync(b->d_plane, 0, 8 * 64, b->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
        if (e != cudaSuccess) st = cuda_fail(e, "batch init", __FILE__, __LINE__);
    }
    if (st != ASC_OK) {
        batch_destroy(b);
        return st;
    }
    *out = b;
    return ASC_OK;
}

bool batch_has_plane(BatchEngine *b, uint32_t slot) { return b->sssp || b->plane[slot] != nullptr; }

// Queues a source for slot (joins before the next iteration). BFS slots need
// their level plane; it is allocated here on first use.
asc_status batch_admit(BatchEngine *b, uint32_t slot, uint32_t source) {
    if (!b->sssp && !b->plane[slot]) {
        ASC_TRY(batch_alloc(b, (void **)&b->plane[slot], 4ull * b->g->V));
        ASC_CUDA(cudaMemcpyAsync(b->d_plane, b->plane, 8 * 64, cudaMemcpyHostToDevice, b->stream));
    }
    b->pend_slot[b->pend_n] = slot;
    b->pend_src[b->pend_n] = source;
    b->pend_n++;
    b->active |= 1ull << slot;
    return ASC_OK;
}

bool batch_busy(const BatchEngine *b) { return b->active != 0; }

// Drops every source of a batch whose launch or collection failed: the batch
// is idle afterwards (its state is undefined until new sources are admitted).
void batch_abort(BatchEngine *b) {
    b->active = 0;
    b->pend_n = 0;
}

uint32_t batch_slots(const BatchEngine *b) { return b->sssp ? b->stride : 64u; }

// Applies the queued admissions and launches one iteration on the batch's
// stream, ending with the readback of its counts (nothing waits here).
namespace {
// Ends a batch iteration: reports the sources still alive to page-locked memory (a
// copy would queue behind the rows that asc_run_batch copies out meanwhile) and
// clears what the next iteration writes, the counts and bitmap that this one read.
__global__ void batch_end_kernel(unsigned long long *alive, unsigned long long *report, uint32_t *cnt,
                                 uint32_t *bitmap, uint32_t nwords) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *report = *alive;
        *alive = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x < CTL_BLOCK) cnt[threadIdx.x] = 0;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) bitmap[w] = 0;
}
}  // namespace

asc_status batch_launch(BatchEngine *b) {
    asc_graph *g = b->g;
    Workspace *ws = &b->ws;
    cudaStream_t s = b->stream;
    const uint32_t V = (uint32_t)g->V;
    const uint32_t nwords = V / 32 + 1;
    const int p = b->parity, po = 1 - p;
    MsArgs m;
    memset(&m, 0, sizeof(m));
    m.front = b->front;
    m.masks = b->masks;
    m.next = b->next;
    m.touched = b->touched;
    m.dist = b->dist;
    m.V = V;
    if (b->pend_n) {
        Admit ad;
        memset(&ad, 0, sizeof(ad));
        ad.n = b->pend_n;
        unsigned long long newmask = 0;
        for (uint32_t i = 0; i < b->pend_n; i++) {
            ad.slot[i] = b->pend_slot[i];
            ad.src[i] = b->pend_src[i];
            newmask |= 1ull << ad.slot[i];
            b->lvl_off[ad.slot[i]] = 2 - (int32_t)(b->it + 1);  // found in the next iteration: level 2
        }
        ASC_CUDA(cudaMemcpyAsync(b->d_lvl_off, b->lvl_off, 4 * 64, cudaMemcpyHostToDevice, s));
        cb_clear_kernel<<<fill_grid(ws, V), kBlock, 0, s>>>(b->masks, b->dist, b->stride, b->d_plane, newmask, V, V + 1,
                                                             b->sssp ? 1 : 0);
        RegionArgs cur = base_args(g, ws, 1 - p);  // the lists/bitmap/counts of parity p (this iteration's input)
        cb_admit_reset_kernel<<<1, 64, 0, s>>>(ad, b->front, ws->bitmap[p]);
        cb_admit_kernel<<<1, 64, 0, s>>>(ad, m, cur, b->d_plane, b->stride, b->sssp ? 1 : 0);
        ASC_CUDA(cudaGetLastError());
        b->pend_n = 0;
    }
    unsigned long long *alive = (unsigned long long *)(ws->ctl + CTL_ALIVE);
    m.r0 = region_args(g, ws, p, 0, false);
    m.r1 = region_args(g, ws, p, 1, false);
    m.work = m.r0.cnt_out + 4;
    if (!b->sssp) {
        attach_items(ws, m.r0);
        attach_items(ws, m.r1);
    }
    const uint32_t grid = (uint32_t)(ws->num_sms * (b->sssp ? ws->tune.ctas_per_sm : ASC_MS_BFS_BLOCKS));
    b->it++;
    if (b->sssp && b->stride == 16) ms_sssp_expand_kernel<16><<<grid, kBlock, 0, s>>>(m);
    else if (b->sssp && b->stride == 32) ms_sssp_expand_kernel<32><<<grid, kBlock, 0, s>>>(m);
    else if (b->sssp) ms_sssp_expand_kernel<64><<<grid, kBlock, 0, s>>>(m);
    else if (g->edge_words == 2) ms_bfs_expand_kernel<2><<<grid, kBlock, 0, s>>>(m);
    else if (g->ebits < 32) ms_bfs_expand_kernel<kBitsLayout><<<grid, kBlock, 0, s>>>(m);
    else ms_bfs_expand_kernel<1><<<grid, kBlock, 0, s>>>(m);
    if (b->sssp) ms_apply_kernel<false><<<fill_grid(ws, 32ull * nwords / kApplyWords), kBlock, 0, s>>>(m, b->d_plane, b->d_lvl_off, b->it,
                                                                               alive, nwords);
    else ms_apply_kernel<true><<<fill_grid(ws, 32ull * nwords / kApplyWords), kBlock, 0, s>>>(m, b->d_plane, b->d_lvl_off, b->it, alive,
                                                                        nwords);
    build_frontier_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(m.r0, ws->bitmap[po], nwords);
    ASC_CUDA(cudaGetLastError());
    batch_end_kernel<<<fill_grid(ws, nwords), kBlock, 0, s>>>(alive, (unsigned long long *)(ws->h_ctl + CTL_ALIVE),
                                                               ws->ctl + CTL_BLOCK * p, ws->bitmap[p], nwords);
    ASC_CUDA(cudaGetLastError());
    b->parity = po;
    return ASC_OK;
}

// Waits for the launched iteration and reports the slots whose sources have
// no frontier left (their values are final).
asc_status batch_collect(BatchEngine *b, uint64_t *finished) {
    ASC_CUDA(cudaStreamSynchronize(b->stream));
    ASC_TRY(self_check_result());
    unsigned long long al = 0;
    memcpy(&al, b->ws.h_ctl + CTL_ALIVE, 8);
    *finished = b->active & ~al;
    b->active &= al;
    return ASC_OK;
}

// Copies a finished slot's values (V u32) to host or device memory.
asc_status batch_fetch(BatchEngine *b, uint32_t slot, void *out, bool device_out = false) {
    const uint32_t V = (uint32_t)b->g->V;
    const cudaMemcpyKind kind = device_out ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    if (b->sssp) {
        cb_gather_column_kernel<<<fill_grid(&b->ws, V), kBlock, 0, b->stream>>>(b->dist, b->stride, slot, b->staging, V);
        ASC_CUDA(cudaGetLastError());
        ASC_CUDA(cudaMemcpyAsync(out, b->staging, 4ull * V, kind, b->stream));
    } else {
        ASC_CUDA(cudaMemcpyAsync(out, b->plane[slot], 4ull * V, kind, b->stream));
    }
    ASC_CUDA(cudaStreamSynchronize(b->stream));
    return ASC_OK;
}

// Makes what copies rows out, before any source runs: nothing of it can fail in
// the middle. Buffers of 64 bytes per vertex that do not fit are done without.
asc_status batch_prepare_rows(BatchEngine *b) {
    if (!b->out_ready) ASC_CUDA(cudaEventCreateWithFlags(&b->out_ready, cudaEventDisableTiming));
    for (auto &s : b->out_stream)
        if (!s) ASC_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    if (!b->sssp || b->out_rows[1]) return ASC_OK;
    asc_status st = ASC_OK;
    for (auto &q : b->out_rows)
        if (st == ASC_OK) st = batch_alloc(b, (void **)&q, 32ull * b->g->V);
    if (st == ASC_OK) return ASC_OK;
    if (b->out_rows[0]) {
        ASC_CUDA(cudaFree(b->out_rows[0]));
        b->out_rows[0] = nullptr;
        b->device_bytes -= 32ull * b->g->V;
    }
    return st == ASC_ERR_BUDGET ? ASC_OK : st;
}

// Starts copying the rows of the finished slots to out (row i of a slot i) on the
// engine's output streams, after what its own stream holds so far: their values
// are final, and later iterations leave them alone. Groups of 8 slots alternate
// between the streams, so the gather of one overlaps the copy of another. Without
// buffers for that, SSSP columns go one at a time through the single column's.
asc_status batch_copy_rows(BatchEngine *b, uint64_t slots, uint32_t *out, bool device_out) {
    const uint64_t V = b->g->V;
    const cudaMemcpyKind kind = device_out ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    ASC_CUDA(cudaEventRecord(b->out_ready, b->stream));
    for (auto s : b->out_stream) ASC_CUDA(cudaStreamWaitEvent(s, b->out_ready, 0));
    if (b->sssp && !b->out_rows[1]) {
        cudaStream_t s = b->out_stream[0];
        for (; slots; slots &= slots - 1) {
            const uint32_t slot = __builtin_ctzll(slots);
            cb_gather_column_kernel<<<fill_grid(&b->ws, V), kBlock, 0, s>>>(b->dist, b->stride, slot, b->staging,
                                                                            (uint32_t)V);
            ASC_CUDA(cudaGetLastError());
            ASC_CUDA(cudaMemcpyAsync(out + slot * V, b->staging, 4 * V, kind, s));
        }
        return ASC_OK;
    }
    for (uint32_t group = 0; group < 8; group++) {
        uint32_t cols = (uint32_t)(slots >> (8 * group)) & 0xffu;
        if (!cols) continue;
        const int i = group & 1;
        cudaStream_t s = b->out_stream[i];
        if (b->sssp) {
            cb_gather_columns_kernel<<<fill_grid(&b->ws, V), kBlock, 0, s>>>(b->dist, b->stride, group, cols,
                                                                              b->out_rows[i], (uint32_t)V);
            ASC_CUDA(cudaGetLastError());
        }
        while (cols) {
            const uint32_t first = __builtin_ctz(cols);
            const uint32_t run = b->sssp ? __builtin_ctz(~(cols >> first)) : 1;  // gathered rows are consecutive
            const uint32_t slot = 8 * group + first;
            ASC_CUDA(cudaMemcpyAsync(out + slot * V, b->sssp ? b->out_rows[i] + first * V : b->plane[slot],
                                     4 * V * run, kind, s));
            cols &= ~(((1u << run) - 1u) << first);
        }
    }
    return ASC_OK;
}

// Waits for the rows on their way out.
cudaError_t batch_finish_rows(BatchEngine *b) {
    cudaError_t first = cudaSuccess;
    for (auto s : b->out_stream) {
        const cudaError_t e = s ? cudaStreamSynchronize(s) : cudaSuccess;
        if (first == cudaSuccess) first = e;
    }
    return first;
}

// run_batch on engine b. After ASC_ERR_TIMEOUT b is empty, after any other error
// its state is undefined; rows may still be on their way out.
static asc_status run_sources(asc_graph *g, BatchEngine *b, const uint32_t *sources, uint32_t n, const asc_params &p,
                              void *out, asc_stats *st) {
    Workspace *ws = g->ws;
    const uint32_t V = (uint32_t)g->V;
    cudaStream_t s = b->stream;
    ASC_CUDA(cudaMemsetAsync(b->ws.ctl + CTL_STATS, 0, 8 * 6, s));
    ASC_CUDA(cudaEventRecord(ws->ev[0], s));
    const bool want = out && !(p.flags & ASC_RUN_NO_OUTPUT);
    if (want) ASC_TRY(batch_prepare_rows(b));
    for (uint32_t i = 0; i < n; i++) ASC_TRY(batch_admit(b, i, sources[i]));
    const uint32_t it0 = b->it;
    const int64_t cap = p.max_iterations > 0 ? p.max_iterations : (int64_t)4 * V + 64;
    std::chrono::steady_clock::time_point done;  // the last iteration's end, on the host
    while (b->active) {
        if ((int64_t)(b->it - it0) >= cap) {
            // drop the unfinished sources so the engine is reusable
            ASC_TRY(batch_clear(b, b->active));
            return fail(ASC_ERR_TIMEOUT, "batch has no fixpoint after %u iterations", b->it - it0);
        }
        uint64_t fin = 0;
        ASC_TRY(batch_launch(b));
        ASC_TRY(batch_collect(b, &fin));
        ASC_CUDA(cudaEventRecord(ws->ev[1], s));
        done = std::chrono::steady_clock::now();
        if (want && fin) ASC_TRY(batch_copy_rows(b, fin, (uint32_t *)out, (p.flags & ASC_RUN_DEVICE_OUT) != 0));
    }
    ASC_CUDA(cudaMemcpyAsync(b->ws.h_ctl + CTL_STATS, b->ws.ctl + CTL_STATS, 8 * 6, cudaMemcpyDeviceToHost, s));
    ASC_CUDA(cudaStreamSynchronize(s));
    ASC_CUDA(batch_finish_rows(b));
    const double copy_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - done).count();
    if (st) {
        memset(st, 0, sizeof(*st));
        const unsigned long long *hs = (const unsigned long long *)(b->ws.h_ctl + CTL_STATS);
        st->iterations = (int32_t)(b->it - it0);
        st->edges_processed = hs[0] + hs[1];
        st->ondemand_edges = hs[1];
        st->ondemand_bytes = edge_store_bytes(g, hs[1]);
        st->frontier_vertices = hs[2] + hs[3];
        st->ondemand_vertices = hs[3];
        float ms = 0;
        ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[0], ws->ev[1]));
        st->ms_total = ms;
        st->ms_copyout = copy_ms;
        st->kernel_launches = (uint32_t)(4 * (b->it - it0) + 3);
    }
    return ASC_OK;
}

// asc_run_batch: all n sources fill slots 0..n-1 of the graph's own batch
// engine (kept for later batches), then iterations run until every source is
// done; each finished slot's values are copied to row i of out. An engine that a
// call left in the middle is not used again: its sources would go on in the next
// call, and their rows are not that call's.
asc_status run_batch(asc_graph *g, asc_algo algo, const uint32_t *sources, uint32_t n, const asc_params &p,
                     void *out, asc_stats *st) {
    ASC_TRY(ensure_workspace(g));
    const int k = algo == ASC_SSSP ? 1 : 0;
    BatchEngine *&b = g->ws->batch[k];
    if (!b) ASC_TRY(batch_create(g, k == 1, 64, &b));
    const asc_status rc = run_sources(g, b, sources, n, p, out, st);
    if (rc == ASC_OK) return rc;
    batch_finish_rows(b);  // no copy into the caller's buffer outlives the call
    if (rc != ASC_ERR_TIMEOUT) {
        batch_destroy(b);
        b = nullptr;
    }
    return rc;
}

// Device bytes of the graph's own batch engines.
uint64_t batch_bytes(const asc_graph *g) {
    uint64_t n = 0;
    if (g->ws)
        for (auto b : g->ws->batch)
            if (b) n += b->device_bytes + b->ws.device_bytes;
    return n;
}

// ------------------------------------------------- PageRank over CSR graphs --
//
// Graphs stored by out-edges (.bcsr / .bwcsr) run PageRank by scatter: every
// vertex adds rank/outDeg to each out-neighbour's sum with an atomic add (FP64
// contributions in FP64; FP32 contributions exactly, as the pull's 62-bit
// fixed point, so an FP32 scatter's sums do not depend on the order of the
// atomics), then one dense pass applies the update. The reference PageRank
// semantics (per-vertex deactivation at |delta| <= 0.001, Jacobi order) and
// the standard ones are the same as the pull kernels'.
namespace {

// Destinations that most edges share, found once per workspace: kPrHot slots by
// a hash of the id, each with the most frequent destination among a sample of
// the edges (count << 32 | id; 0: empty). Their atomics meet in a few L2 slices:
// on 1 M RMAT vertices the busiest slice took 451,000 of the pass's atomic
// sectors against 128,000 on average, and set the pass's time (24 passes of 16 M
// edges: 8.20 ms without the slots; 4.36 / 4.18 / 4.15 / 4.20 ms with 256 / 512 /
// 1024 / 2048, the last two at 4 CTAs per SM, 4.29 with 1024 at 6; tiles of 256
// vertices instead of items: 9.53 ms).
constexpr uint32_t kPrHotSample = 16;   // every how many items are sampled
__device__ __forceinline__ uint32_t pr_hot_slot(uint32_t v) { return (v * 2654435761u) >> (32 - __ffs(kPrHot) + 1); }

template <typename T>
__global__ void pr_hot_count_kernel(PrItemArgs<T> p, unsigned long long *count) {
    const uint32_t mask = p.ebits >= 32 ? 0xffffffffu : (1u << p.ebits) - 1u;
    const uint32_t total = p.sl[0].n + p.sl[1].n;
    for (uint32_t it = blockIdx.x * kPrHotSample; it < total; it += gridDim.x * kPrHotSample) {
        const PrSlice &sl = p.sl[it >= p.sl[0].n];
        const uint32_t e0 = p.items[it].y, e1 = p.items[it + 1].y;
        for (uint32_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
            const uint64_t bit = (uint64_t)e * p.ebits;
            const uint64_t w = bit >> 5;
            const uint32_t hi = w + 1 < sl.edge_words ? __ldg(sl.edges + w + 1) : 0u;
            const uint32_t v = (__funnelshift_r(__ldg(sl.edges + w), hi, (uint32_t)bit & 31u) & mask) >> p.wbits;
            if (!ASC_BAD(v >= p.V, 18, v)) atomicAdd(&count[v], 1ull);
        }
    }
}

// Puts the counts into the slots and clears them.
__global__ void pr_hot_pick_kernel(unsigned long long *count, uint32_t V, unsigned long long *slots) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const unsigned long long n = count[v];
        if (!n) continue;
        count[v] = 0;
        unsigned long long *s = slots + pr_hot_slot(v);
        const unsigned long long x = (n << 32) | v;
        if (*s < x) atomicMax(s, x);
    }
}

// A CTA's sums of the hot destinations.
template <typename T>
struct PrHot;
template <>
struct PrHot<double> {
    uint32_t key[kPrHot];
    double acc[kPrHot];
    __device__ __forceinline__ void clear(uint32_t i) { acc[i] = 0; }
    __device__ __forceinline__ void add(uint32_t i, double x) { atomicAdd(&acc[i], x); }
    __device__ __forceinline__ double get(uint32_t i) const { return acc[i]; }
};
template <>
struct PrHot<float> {
    uint32_t key[kPrHot];
    uint32_t lo[kPrHot], hi[kPrHot];  // 64-bit fixed point as two 32-bit shared atomics with the carry between
    __device__ __forceinline__ void clear(uint32_t i) { lo[i] = hi[i] = 0; }
    __device__ __forceinline__ void add(uint32_t i, unsigned long long x) {
        const uint32_t xl = (uint32_t)x, old = atomicAdd(&lo[i], xl);
        const uint32_t xh = (uint32_t)(x >> 32) + (old + xl < xl ? 1u : 0u);
        if (xh) atomicAdd(&hi[i], xh);
    }
    __device__ __forceinline__ unsigned long long get(uint32_t i) const {
        return ((unsigned long long)hi[i] << 32) | lo[i];
    }
};

// Edge-balanced scatter: items as in pr_pull_items_kernel, over out-edges. The
// contributions of the item's rows are converted once into shared memory; a
// thread adds its row's to the destinations of kVt consecutive edges, passing
// to the next row at each mark. Hot destinations add up in shared memory and
// reach the global sums once per CTA; the rest are atomics in L2, which bound
// the pass. wbits > 0: edge words hold the weight below the destination; ebits
// 64: {dst, weight}.
template <typename T>
__global__ void __launch_bounds__(kBlock, ASC_PR_SCATTER_BLOCKS) pr_scatter_items_kernel(PrItemArgs<T> p) {
    typedef typename PrAcc<T>::type Acc;
    if (p.active_prev ? !*p.active_prev : pr_pass_over<false>(p)) return;
    __shared__ PrItemSmem<T> sm;
    __shared__ PrHot<T> hot;
    for (uint32_t i = threadIdx.x; i < kPrHot; i += kBlock) {
        const unsigned long long x = p.hot[i];
        hot.key[i] = x ? (uint32_t)x : 0xffffffffu;
        hot.clear(i);
    }
    const int lane = threadIdx.x & 31;
    const uint32_t total = p.sl[0].n + p.sl[1].n;
    const uint32_t eb = p.ebits, mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
    if (threadIdx.x < kItem / 32) sm.marks[0][threadIdx.x] = sm.marks[1][threadIdx.x] = 0;
    if (threadIdx.x == 0) sm.work[0] = atomicAdd(p.work, 1u);
    __syncthreads();
    for (int buf = 0;; buf ^= 1) {
        const uint32_t w = sm.work[buf];
        if (w >= total) break;
        bool od;
        const uint32_t it = pr_slice_item(p.sl, w, od);
        const uint2 a = p.items[it], b = p.items[it + 1];
        const uint32_t r0 = a.x, e0 = a.y, nr = b.x - a.x, ne = b.y - a.y;
        uint32_t nq;
        const uint32_t bit0 = stage_words(p.sl[od].edges, p.sl[od].edge_words, e0, ne, eb, sm.pool, nq);
        Acc *share = reinterpret_cast<Acc *>(sm.pool + 4 * nq + (nq ? 4 : 0));
        for (uint32_t j = threadIdx.x; j <= nr; j += kBlock)
            share[j] = r0 + j < p.V ? PrAcc<T>::from(p.c_old[r0 + j]) : (Acc)0;
        uint32_t *marks = sm.marks[buf];
        pr_mark_rows<T>(p.ptr, r0, e0, nr, sm, marks);
        if (threadIdx.x == 0) sm.work[buf ^ 1] = atomicAdd(p.work, 1u);
        __syncthreads();
        if (threadIdx.x < kItem / 32) sm.marks[buf ^ 1][threadIdx.x] = 0;
        const uint32_t x0 = threadIdx.x * kVt, xw = x0 - lane * kVt;
        if (xw < ne) {
            const uint32_t ends = (marks[x0 >> 5] >> (x0 & 31)) & ((1u << kVt) - 1u);
            // the row that is open after this thread's edges: of the next mark in
            // a later lane, in a later warp, or the one that goes on past the item
            const unsigned ended = __ballot_sync(kFull, ends != 0);
            const uint32_t first = ends ? sm.row_at[x0 + __ffs((int)ends) - 1] : nr;
            const unsigned above = lane < 31 ? ended & (0xffffffffu << (lane + 1)) : 0u;
            const uint32_t from_lane = __shfl_sync(kFull, first, above ? __ffs((int)above) - 1 : lane);
            const uint32_t after = pr_next_row(marks, sm.row_at, xw + 32 * kVt, nr);
            const uint32_t open = above ? from_lane : after;
            Acc c = share[ends ? first : open];
            uint32_t v[kVt];
#pragma unroll
            for (int k = 0; k < kVt; k++)
                v[k] = x0 + k < ne ? staged_word(sm.pool, bit0 + (x0 + k) * eb, mask) >> p.wbits : 0u;
            // Consecutive edges to one destination (the leaves of a hub, duplicates) are
            // one add: FP64 adds to one shared address go one after the other (1,000 hubs
            // of 2,000 leaves: 28.1 ms an add per edge, 12.1 so). A warp without any skips
            // the comparisons, which cost 3 to 5% of an FP64 pass on other graphs.
            bool same = false;
#pragma unroll
            for (int k = 1; k < kVt; k++) same = same || (v[k] == v[k - 1] && x0 + k < ne);
            const bool runs = __any_sync(kFull, same);
            auto add = [&](uint32_t to, Acc x) {
                const uint32_t h = pr_hot_slot(to);
                if (hot.key[h] == to) hot.add(h, x);
                else atomicAdd(&p.sum[to], x);
            };
            auto next_row = [&](int k) {
                if (!((ends >> k) & 1u)) return;
                const uint32_t rest = ends >> k >> 1;
                c = share[rest ? sm.row_at[x0 + k + __ffs((int)rest)] : open];
            };
            if (!runs) {
#pragma unroll
                for (int k = 0; k < kVt; k++) {
                    if (x0 + k < ne && !ASC_BAD(v[k] >= p.V, 18, v[k])) add(v[k], c);
                    next_row(k);
                }
            } else {
                Acc run = (Acc)0;
#pragma unroll
                for (int k = 0; k < kVt; k++) {
                    if (x0 + k < ne && !ASC_BAD(v[k] >= p.V, 18, v[k])) {
                        run += c;
                        if (k + 1 == kVt || x0 + k + 1 >= ne || v[k + 1 < kVt ? k + 1 : k] != v[k]) {
                            add(v[k], run);
                            run = (Acc)0;
                        }
                    }
                    next_row(k);
                }
            }
        }
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < kPrHot; i += kBlock) {
        const Acc x = hot.get(i);
        if (x != (Acc)0) atomicAdd(&p.sum[hot.key[i]], x);
    }
}

// The update of every vertex after a scatter; ends the pass. Reference mode:
// active holds one bit per vertex that is still active, active_count this
// pass's and active_next the next one's number of them.
template <typename T, bool REF>
__global__ void __launch_bounds__(kBlock) pr_push_apply_kernel(PrItemArgs<T> p, uint32_t *active,
                                                                   uint32_t *active_count, uint32_t *active_next) {
    if (p.active_prev ? !*p.active_prev : pr_pass_over<false>(p)) return;
    __shared__ double red[2 * kWarps];
    __shared__ double s_base;
    const uint32_t V = p.V;
    if (!REF) {
        if (threadIdx.x == 0) s_base = (1.0 - p.damping) / (double)V + p.damping * (*p.dangling_prev) / (double)V;
        __syncthreads();
    }
    double res = 0, dang = 0;
    uint32_t nact = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const double s = PrAcc<T>::value(p.sum[v]);
        p.sum[v] = 0;
        const uint32_t od = p.ptr[v + 1] - p.ptr[v];
        if (REF) {
            const uint32_t bit = 1u << (v & 31);
            if (!(active[v >> 5] & bit)) {
                p.c_new[v] = p.c_old[v];
                continue;
            }
            if (pr_ref_row((double *)p.rank, (const double *)p.c_old, (double *)p.c_new, v, od, s)) nact++;
            else atomicAnd(&active[v >> 5], ~bit);
        } else {
            pr_std_row<T>(p.rank, p.c_new, v, od, s, p.damping, s_base, res, dang);
        }
    }
    if (!REF) {
        block_reduce2_atomic(res, dang, p.acc, red);
        pr_end_pass<false>(p);
        return;
    }
    nact = __reduce_add_sync(kFull, nact);
    if ((threadIdx.x & 31) == 0 && nact) atomicAdd(active_count, nact);
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(p.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last || threadIdx.x) return;
    __threadfence();
    *(volatile unsigned long long *)p.report = *(volatile uint32_t *)active_count;
    *active_next = 0;
    *p.work = 0;
    *p.ticket = 0;
}

template <typename T>
__global__ void pr_push_init_kernel(double *rank, T *c0, T *c1, typename PrAcc<T>::type *sum, const uint32_t *ptr,
                                    uint32_t *active, uint32_t V, double *acc_pair) {
    __shared__ double red[2 * kWarps];
    double d = 0;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < V; base += stride) {
        const uint32_t i = base + threadIdx.x;
        if (i < V) {
            const double r = 1.0 / (double)V;
            const uint32_t od = ptr[i + 1] - ptr[i];
            rank[i] = r;
            const T c = od ? (T)(r / (double)od) : (T)0;
            c0[i] = c;
            c1[i] = c;
            sum[i] = 0;
            if (od == 0) d += r;
        }
        if (i < (V + 31) / 32) active[i] = 0xffffffffu;
    }
    block_reduce2_atomic(0.0, d, acc_pair, red);
}

}  // namespace

template <typename T, bool REF, int WORDS>
static asc_status pagerank_push_impl(asc_graph *g, const asc_params &p, void *out, asc_stats *st) {
    Workspace *ws = g->ws;
    ASC_TRY(ensure_pr_buffers(g, sizeof(T)));
    const uint32_t V = (uint32_t)g->V;
    cudaStream_t s = g->stream;
    uint32_t launches = 0;
    typedef typename PrAcc<T>::type Acc;
    double *rank = (double *)ws->pr_rank;
    T *c[2] = {(T *)ws->pr_contrib[0], (T *)ws->pr_contrib[1]};
    uint32_t *active = ws->bitmap[1];

    ASC_CUDA(cudaEventRecord(ws->ev[0], s));
    ASC_CUDA(cudaMemsetAsync(ws->ctl, 0, 4 * CTL_WORDS, s));
    pr_push_init_kernel<T><<<fill_grid(ws, V), kBlock, 0, s>>>(rank, c[0], c[1], (Acc *)ws->pr_sum, g->d_ptr, active,
                                                               V, (double *)(ws->ctl + CTL_ACC) + 4);
    launches++;
    bool staged = false;
    if (!REF && !(p.flags & ASC_RUN_NO_STAGING)) ASC_TRY(ensure_stage_plan(g, &staged));
    ASC_CUDA(cudaGetLastError());
    const int max_it = p.max_iterations > 0 ? p.max_iterations : (REF ? 1000000 : 100);
    StagePlan *sp = staged ? ws->stage : nullptr;
    PrItemArgs<T> ia;
    memset(&ia, 0, sizeof(ia));
    ASC_TRY(ensure_items(g));
    ia.items = ws->items;
    ia.sl[0] = pr_slice(g, 0);
    ia.sl[1] = pr_slice(g, 1);
    ia.ptr = g->d_ptr;
    ia.sum = (Acc *)ws->pr_sum;
    ia.rank = rank;
    ia.cnt_in = ws->ctl + CTL_BLOCK;
    ia.work = ws->ctl + CTL_BLOCK + 4;
    ia.V = V;
    ia.ebits = WORDS == 2 ? 64 : g->ebits;
    ia.wbits = g->wbits;
    if (!ws->pr_hot) {
        ASC_CUDA(cudaMalloc((void **)&ws->pr_hot, 8 * kPrHot));
        ws->device_bytes += 8 * kPrHot;
        ASC_CUDA(cudaMemsetAsync(ws->pr_hot, 0, 8 * kPrHot, s));
        pr_hot_count_kernel<T><<<item_grid(ws, ws->n_items / kPrHotSample + 1, 8), kBlock, 0, s>>>(
            ia, (unsigned long long *)ws->pr_sum);
        pr_hot_pick_kernel<<<fill_grid(ws, V), kBlock, 0, s>>>((unsigned long long *)ws->pr_sum, V, ws->pr_hot);
        launches += 2;
        ASC_CUDA(cudaGetLastError());
    }
    ia.hot = ws->pr_hot;
    ASC_TRY(ensure_pass_events(ws));
    const int depth = staged || t_iteration_hook.fn ? 1 : 2;
    int it = 0, launched = 0;  // passes that ended, that were launched
    double residual = 0;
    bool over = false;
    for (;;) {
        if (launched - it >= depth || (launched > it && launched >= max_it)) {
            ASC_CUDA(cudaEventSynchronize(ws->pass_ev[it % kPassSlots]));
            const unsigned long long *r = pass_slot(ws, it);
            memcpy(&residual, r, 8);
            over = REF ? r[0] == 0 : residual < p.tolerance;
            if (REF) residual = 0;
            it++;
            iteration_boundary();
        }
        if (over) break;  // a pass launched after the last one changes nothing
        if (launched >= max_it) {
            if (launched > it) continue;
            if (REF) return fail(ASC_ERR_TIMEOUT, "reference PageRank still active after %d passes", it);
            break;
        }
        ia.c_old = c[launched & 1];
        ia.c_new = c[1 - (launched & 1)];
        set_pass(ws, p, launched, ia);
        uint32_t *counts = ws->ctl + CTL_PR;  // reference mode: active vertices after three consecutive passes
        ia.active_prev = REF && launched ? counts + (launched + 2) % 3 : nullptr;
        if (staged) ASC_CUDA(cudaMemsetAsync(sp->d_work, 0, 4 * sp->launches.size(), s));
        for (uint32_t k = 0; k < (staged ? (uint32_t)sp->launches.size() : 1u); k++) {
            if (staged) {
                ASC_TRY(stage_chunk(g, sp, k, s, ia.sl));
                ia.work = sp->d_work + k;
            }
            pr_scatter_items_kernel<T><<<item_grid(ws, ia.sl[0].n + ia.sl[1].n, ASC_PR_SCATTER_BLOCKS), kBlock, 0,
                                         s>>>(ia);
            if (staged) ASC_TRY(stage_release(sp, k, s));
            launches++;
        }
        pr_push_apply_kernel<T, REF><<<fill_grid(ws, V), kBlock, 0, s>>>(ia, active, counts + launched % 3,
                                                                              counts + (launched + 1) % 3);
        launches++;
        ASC_CUDA(cudaGetLastError());
        ASC_CUDA(cudaEventRecord(ws->pass_ev[launched % kPassSlots], s));
        launched++;
    }
    ASC_CUDA(cudaEventRecord(ws->ev[1], s));
    if (out && !(p.flags & ASC_RUN_NO_OUTPUT)) {
        ASC_TRY(copy_ranks_out<T>(g, rank, (void *)c[0], out, p.flags));
        launches += sizeof(T) == 4;
    }
    ASC_CUDA(cudaEventRecord(ws->ev[2], s));
    ASC_CUDA(cudaStreamSynchronize(s));
    if (st) {
        memset(st, 0, sizeof(*st));
        unsigned long long n[4];
        pr_pass_counts(g, (uint64_t)it, n);
        st->iterations = it;
        st->edges_processed = n[0] + n[1];
        st->ondemand_edges = n[1];
        st->ondemand_bytes = staged ? sp->copy_bytes * (uint64_t)it : edge_store_bytes(g, n[1]);
        st->staged_chunks = staged ? (uint32_t)(sp->launches.size() * it) : 0;
        st->frontier_vertices = n[2] + n[3];
        st->ondemand_vertices = n[3];
        st->reached_vertices = V;
        st->reached_edges = g->E;
        st->residual = residual;
        float ms = 0;
        ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[0], ws->ev[1]));
        st->ms_total = ms;
        ASC_CUDA(cudaEventElapsedTime(&ms, ws->ev[1], ws->ev[2]));
        st->ms_copyout = ms;
        st->kernel_launches = launches;
    }
    return ASC_OK;
}

asc_status run_pagerank(asc_graph *g, const asc_params &p, void *out, asc_stats *st) {
    ASC_TRY(ensure_workspace(g));
    if (!g->is_csc) {
        const bool w2 = g->edge_words == 2;
        if (p.pr_mode == ASC_PR_REF)
            return w2 ? pagerank_push_impl<double, true, 2>(g, p, out, st)
                      : pagerank_push_impl<double, true, 1>(g, p, out, st);
        if (p.precision == ASC_F32)
            return w2 ? pagerank_push_impl<float, false, 2>(g, p, out, st)
                      : pagerank_push_impl<float, false, 1>(g, p, out, st);
        return w2 ? pagerank_push_impl<double, false, 2>(g, p, out, st)
                  : pagerank_push_impl<double, false, 1>(g, p, out, st);
    }
    if (p.pr_mode == ASC_PR_REF) return pagerank_impl<double, true>(g, p, out, st);
    if (p.precision == ASC_F32) return pagerank_impl<float, false>(g, p, out, st);
    return pagerank_impl<double, false>(g, p, out, st);
}

}  // namespace asc

namespace {
__global__ void link_read_kernel(const uint4 *__restrict__ src, size_t n16, unsigned long long *sink) {
    // four independent 16-byte loads in flight per thread
    uint32_t acc = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n16; i += 4 * stride) {
        uint4 a = __ldg(src + i), b = __ldg(src + i + stride), c = __ldg(src + i + 2 * stride),
              d = __ldg(src + i + 3 * stride);
        acc ^= a.x ^ a.y ^ a.z ^ a.w ^ b.x ^ b.y ^ b.z ^ b.w ^ c.x ^ c.y ^ c.z ^ c.w ^ d.x ^ d.y ^ d.z ^ d.w;
    }
    for (; i < n16; i += stride) {
        uint4 v = __ldg(src + i);
        acc ^= v.x ^ v.y ^ v.z ^ v.w;
    }
    if (acc == 0x9e3779b9u) atomicAdd(sink, 1ull);  // keeps the loads live
}
__device__ __forceinline__ uint64_t probe_mix(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    return x ^ (x >> 33);
}

// Each warp reads `runs` runs of L consecutive words at pseudo-random word
// offsets in [0, n4 - L), four runs in flight, lanes striding the run: the
// access shape of short adjacency lists read over the host link.
__global__ void link_runs_kernel(const uint32_t *__restrict__ src, uint64_t n4, uint32_t L, uint32_t runs,
                                 unsigned long long *sink) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t acc = 0;
    for (uint32_t r = 0; r < runs; r += 4) {
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t off = probe_mix(warp * 1000003ull + r + k) % (n4 - L);  // off + L < n4
            v[k] = 0;
            for (uint32_t j = lane; j < L; j += 32) v[k] ^= __ldg(src + off + j);
        }
        acc ^= v[0] ^ v[1] ^ v[2] ^ v[3];
    }
    if (acc == 0x9e3779b9u) atomicAdd(sink, 1ull);  // keeps the loads live
}
}  // namespace

extern "C" asc_status asc_link_probe_runs(uint64_t bytes, uint32_t run_bytes, int iters, double *gbs) {
    using namespace asc;
    if (bytes < (1u << 20) || iters < 1 || run_bytes < 4 || run_bytes % 4 || run_bytes > bytes / 16)
        return fail(ASC_ERR_INVALID, "asc_link_probe_runs: bytes >= 1 MiB, 4 <= run_bytes <= bytes/16, "
                                     "run_bytes a multiple of 4, iters >= 1");
    bytes &= ~(uint64_t)15;
    void *h = nullptr, *hd = nullptr;
    unsigned long long *sink = nullptr;
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    asc_status st = ASC_OK;
    double best = 0;
    int sms = 0, dev = 0;
    auto chk = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && st == ASC_OK) st = cuda_fail(e, what, __FILE__, __LINE__);
        return st == ASC_OK;
    };
    if (chk(cudaHostAlloc(&h, bytes, cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc") &&
        chk(cudaHostGetDevicePointer(&hd, h, 0), "cudaHostGetDevicePointer") &&
        chk(cudaMalloc(&sink, 8), "cudaMalloc") && chk(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream") &&
        chk(cudaEventCreate(&e0), "event") && chk(cudaEventCreate(&e1), "event") && chk(cudaGetDevice(&dev), "dev") &&
        chk(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr")) {
        memset(h, 1, bytes);
        const uint64_t n4 = bytes / 4;
        const uint32_t L = run_bytes / 4;
        const uint64_t warps = (uint64_t)sms * 8 * (256 / 32);
        // about one pass over the buffer, a multiple of 4 runs per warp
        const uint32_t runs = (uint32_t)std::max<uint64_t>(4, (n4 / (warps * L)) & ~3ull);
        for (int i = 0; i < iters + 1 && st == ASC_OK; i++) {
            float ms = 0;
            chk(cudaEventRecord(e0, s), "rec");
            link_runs_kernel<<<sms * 8, 256, 0, s>>>((const uint32_t *)hd, n4, L, runs, sink);
            chk(cudaGetLastError(), "launch");
            chk(cudaEventRecord(e1, s), "rec");
            chk(cudaEventSynchronize(e1), "sync");
            chk(cudaEventElapsedTime(&ms, e0, e1), "elapsed");
            if (i > 0 && ms > 0) best = std::max(best, (double)warps * runs * run_bytes / (ms * 1e6));
        }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (s) cudaStreamDestroy(s);
    if (sink) cudaFree(sink);
    if (h) cudaFreeHost(h);
    if (gbs) *gbs = best;
    return st;
}

extern "C" asc_status asc_link_probe(uint64_t bytes, int iters, double *dma_h2d_gbs, double *sm_read_gbs) {
    using namespace asc;
    if (bytes < (1u << 20) || iters < 1) return fail(ASC_ERR_INVALID, "asc_link_probe: bytes >= 1 MiB, iters >= 1");
    bytes &= ~(uint64_t)15;
    void *h = nullptr, *d = nullptr, *hd = nullptr;
    unsigned long long *sink = nullptr;
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    asc_status st = ASC_OK;
    double best_dma = 0, best_sm = 0;
    int sms = 0, dev = 0;
    auto chk = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && st == ASC_OK) st = cuda_fail(e, what, __FILE__, __LINE__);
        return st == ASC_OK;
    };
    if (chk(cudaHostAlloc(&h, bytes, cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc") &&
        chk(cudaHostGetDevicePointer(&hd, h, 0), "cudaHostGetDevicePointer") &&
        chk(cudaMalloc(&d, bytes), "cudaMalloc") && chk(cudaMalloc(&sink, 8), "cudaMalloc") &&
        chk(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream") &&
        chk(cudaEventCreate(&e0), "event") && chk(cudaEventCreate(&e1), "event") &&
        chk(cudaGetDevice(&dev), "dev") &&
        chk(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr")) {
        memset(h, 1, bytes);
        for (int i = 0; i < iters + 1 && st == ASC_OK; i++) {
            // one copy per quarter, issued back to back on one stream
            float ms = 0;
            chk(cudaEventRecord(e0, s), "rec");
            const uint64_t q = (bytes / 4) & ~(uint64_t)15;
            for (int k = 0; k < 4; k++) {
                uint64_t off = k * q, n = k == 3 ? bytes - off : q;
                chk(cudaMemcpyAsync((char *)d + off, (const char *)h + off, n, cudaMemcpyHostToDevice, s),
                    "memcpy");
            }
            chk(cudaEventRecord(e1, s), "rec");
            chk(cudaEventSynchronize(e1), "sync");
            chk(cudaEventElapsedTime(&ms, e0, e1), "elapsed");
            if (i > 0 && ms > 0) best_dma = std::max(best_dma, bytes / (ms * 1e6));
        }
        for (int i = 0; i < iters + 1 && st == ASC_OK; i++) {
            float ms = 0;
            chk(cudaEventRecord(e0, s), "rec");
            link_read_kernel<<<sms * 16, 256, 0, s>>>((const uint4 *)hd, bytes / 16, sink);
            chk(cudaGetLastError(), "launch");
            chk(cudaEventRecord(e1, s), "rec");
            chk(cudaEventSynchronize(e1), "sync");
            chk(cudaEventElapsedTime(&ms, e0, e1), "elapsed");
            if (i > 0 && ms > 0) best_sm = std::max(best_sm, bytes / (ms * 1e6));
        }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (s) cudaStreamDestroy(s);
    if (sink) cudaFree(sink);
    if (d) cudaFree(d);
    if (h) cudaFreeHost(h);
    if (dma_h2d_gbs) *dma_h2d_gbs = best_dma;
    if (sm_read_gbs) *sm_read_gbs = best_sm;
    return st;
}

// ------------------------------------------------- allocation-free BFS -------
//
// asc_bfs_device_noalloc runs the same BFS expansion kernel over a CSR graph the
// caller already holds in device memory, for callers that cannot allocate
// device memory at query time: a process whose device memory is owned by
// another allocator (a framework's caching pool sized to the whole GPU, where
// a cudaMalloc of its own would fail or fragment the pool), or a latency-bound
// loop where cudaMalloc/cudaFree (which can synchronize the device) are not
// allowed. Its scratch state (frontier lists, segment lists, the next-frontier
// bitmap, counters) lives in one file-scope device array of fixed size, which
// every GPU that loads this library holds until the process exits.
namespace asc {
namespace {

constexpr uint64_t kNoAllocMaxV = 1ull << 20;   // vertices
constexpr uint64_t kNoAllocMaxE = 1ull << 24;   // edges
constexpr uint32_t kNoAllocHuge = 512;          // same degree buckets as the default Tuning
constexpr uint32_t kNoAllocSeg = 2048;
// segment items never exceed E/seg_len (full segments) + E/huge (one partial per long list)
constexpr uint64_t kNoAllocMaxSegs = kNoAllocMaxE / kNoAllocSeg + kNoAllocMaxE / kNoAllocHuge + 1;

constexpr uint64_t na_round(uint64_t x) { return (x + 255) & ~255ull; }
constexpr uint64_t kNaCtl = 0;
constexpr uint64_t kNaBitmap = na_round(kNaCtl + 4 * CTL_WORDS);
constexpr uint64_t kNaBitmap1 = na_round(kNaBitmap + 4 * (kNoAllocMaxV / 32 + 2));
constexpr uint64_t kNaVisited = na_round(kNaBitmap1 + 4 * (kNoAllocMaxV / 32 + 2));
constexpr uint64_t kNaHuge = na_round(kNaVisited + 4 * (kNoAllocMaxV / 32 + 2));
constexpr uint64_t kNaQueue0 = na_round(kNaHuge + 4 * (kNoAllocMaxV / 32 + 2));
constexpr uint64_t kNaQueue1 = na_round(kNaQueue0 + 4 * kNoAllocMaxV);
constexpr uint64_t kNaSegs0 = na_round(kNaQueue1 + 4 * kNoAllocMaxV);
constexpr uint64_t kNaSegs1 = na_round(kNaSegs0 + 8 * kNoAllocMaxSegs);
constexpr uint64_t kNaBytes = na_round(kNaSegs1 + 8 * kNoAllocMaxSegs);   // about 9.6 MB

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

// In host code g_noalloc_scratch names a host-side stand-in, not device memory;
// kernels get the device address looked up once per device. The cached address
// belongs to the device's primary context: a cudaDeviceReset or another context
// would leave it stale, which the header rules out for callers.
constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
unsigned char *g_na_addr[kNaMaxDevices] = {nullptr};

// Checks the caller's CSR on the device: offsets start at 0, never decrease,
// end at E, destinations are < V. flag[0] becomes nonzero on the first defect.
__global__ void noalloc_validate_kernel(const uint32_t *ptr, const uint32_t *col, uint32_t V, uint32_t E,
                                        uint32_t *flag) {
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0 && (ptr[0] != 0 || ptr[V] != E)) atomicOr(flag, 1u);
    for (uint32_t v = t; v < V; v += stride)
        if (ptr[v] > ptr[v + 1]) atomicOr(flag, 2u);
    for (uint32_t i = t; i < E; i += stride)
        if (col[i] >= V) atomicOr(flag, 4u);
}

// One bit per vertex whose list is longer than the huge-degree threshold.
__global__ void noalloc_huge_bits_kernel(const uint32_t *ptr, uint32_t V, uint32_t huge, uint32_t *bits,
                                         uint32_t nwords) {
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
        uint32_t m = 0;
        for (uint32_t b = 0; b < 32; b++) {
            const uint32_t v = 32 * w + b;
            if (v < V && ptr[v + 1] - ptr[v] > huge) m |= 1u << b;
        }
        bits[w] = m;
    }
}

asc_status noalloc_scratch(unsigned char **out) {
    int dev = 0;
    ASC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNaMaxDevices) return fail(ASC_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!g_na_addr[dev]) {
        void *p = nullptr;
        ASC_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_na_addr[dev] = (unsigned char *)p;
    }
    *out = g_na_addr[dev];
    return ASC_OK;
}

}  // namespace
}  // namespace asc

extern "C" asc_status asc_bfs_device_noalloc(uint64_t V, uint64_t E, const uint32_t *d_row_offsets,
                                             const uint32_t *d_col, uint32_t source, uint32_t *d_levels,
                                             void *stream) {
    using namespace asc;
    if (!d_row_offsets || !d_levels || (!d_col && E))
        return fail(ASC_ERR_INVALID, "asc_bfs_device_noalloc: null device pointer");
    if (V == 0 || V > kNoAllocMaxV)
        return fail(ASC_ERR_BUDGET, "asc_bfs_device_noalloc: V = %llu outside [1, %llu], the fixed scratch limit",
                    (unsigned long long)V, (unsigned long long)kNoAllocMaxV);
    if (E > kNoAllocMaxE)
        return fail(ASC_ERR_BUDGET, "asc_bfs_device_noalloc: E = %llu above %llu, the fixed scratch limit",
                    (unsigned long long)E, (unsigned long long)kNoAllocMaxE);
    if (source >= V) return fail(ASC_ERR_INVALID, "source %u is not a vertex (V = %llu)", source,
                                 (unsigned long long)V);
    unsigned char *base = nullptr;
    ASC_TRY(noalloc_scratch(&base));
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t *ctl = (uint32_t *)(base + kNaCtl);
    uint32_t *bitmap[2] = {(uint32_t *)(base + kNaBitmap), (uint32_t *)(base + kNaBitmap1)};
    uint32_t *visited = (uint32_t *)(base + kNaVisited);
    uint32_t *huge_bits = (uint32_t *)(base + kNaHuge);
    uint32_t *queue[2] = {(uint32_t *)(base + kNaQueue0), (uint32_t *)(base + kNaQueue1)};
    uint64_t *segs[2] = {(uint64_t *)(base + kNaSegs0), (uint64_t *)(base + kNaSegs1)};
    const uint32_t V32 = (uint32_t)V, E32 = (uint32_t)E;
    const uint32_t nwords = V32 / 32 + 1;
    int dev = 0, sms = 0;
    ASC_CUDA(cudaGetDevice(&dev));
    ASC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint32_t fill = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((V + kBlock - 1) / kBlock, sms * 8ull));

    // the array keeps the previous call's contents: clear the counters and the
    // bitmaps first
    ASC_CUDA(cudaMemsetAsync(ctl, 0, 4 * CTL_WORDS, s));
    ASC_CUDA(cudaMemsetAsync(visited, 0, 4 * (V / 32 + 2), s));
    for (int i = 0; i < 2; i++) ASC_CUDA(cudaMemsetAsync(bitmap[i], 0, 4 * (V / 32 + 2), s));
    noalloc_validate_kernel<<<fill, kBlock, 0, s>>>(d_row_offsets, d_col, V32, E32, ctl + CTL_PR);
    ASC_CUDA(cudaGetLastError());
    uint32_t flag = 0;
    ASC_CUDA(cudaMemcpyAsync(&flag, ctl + CTL_PR, 4, cudaMemcpyDeviceToHost, s));
    ASC_CUDA(cudaStreamSynchronize(s));
    if (flag)
        return fail(ASC_ERR_INVALID, "asc_bfs_device_noalloc: malformed CSR (%s%s%s)",
                    flag & 1 ? "offsets must start at 0 and end at E; " : "",
                    flag & 2 ? "offsets decrease; " : "", flag & 4 ? "destination >= V" : "");
    noalloc_huge_bits_kernel<<<fill, kBlock, 0, s>>>(d_row_offsets, V32, kNoAllocHuge, huge_bits, nwords);

    RegionArgs a;
    memset(&a, 0, sizeof(a));
    a.ptr = d_row_offsets;
    a.edges = d_col;
    a.ebits = 32;
    a.val = d_levels;
    a.visited = visited;
    a.huge_bits = huge_bits;
    a.S = V32;  // the whole graph is device resident: one region
    a.V = V32;
    a.dense_begin = 0;
    a.dense_end = V32;
    a.dense_div = 64;
    a.huge = kNoAllocHuge;
    a.seg_len = kNoAllocSeg;
    a.segcap_static = (uint32_t)kNoAllocMaxSegs;
    a.stats = (unsigned long long *)(ctl + CTL_STATS);
    // seed: the source lands in parity 0
    a.cnt_out = ctl;
    a.q_out = queue[0];
    a.seg_out = segs[0];
    a.bitmap = bitmap[0];
    init_values_kernel<kBFS><<<fill, kBlock, 0, s>>>(d_levels, V32, source);
    seed_bits_kernel<<<1, kBlock, 0, s>>>(a, source, 0, nwords);
    build_frontier_kernel<<<fill, kBlock, 0, s>>>(a, bitmap[0], nwords);
    ASC_CUDA(cudaGetLastError());
    uint32_t cnt[CTL_BLOCK] = {0, 0, 0, 0, 0, 0, 0, 0};
    ASC_CUDA(cudaMemcpyAsync(cnt, ctl, sizeof(cnt), cudaMemcpyDeviceToHost, s));
    ASC_CUDA(cudaStreamSynchronize(s));
    int parity = 0;
    int64_t iters = 0;
    while (cnt[6] | cnt[7]) {
        if (++iters > (int64_t)V + 2) return fail(ASC_ERR_TIMEOUT, "no fixpoint after %lld iterations",
                                                  (long long)iters);
        const int po = 1 - parity;
        ASC_CUDA(cudaMemsetAsync(ctl + CTL_BLOCK * po, 0, 4 * CTL_BLOCK, s));
        ASC_CUDA(cudaMemsetAsync(bitmap[po], 0, 4 * (V / 32 + 2), s));
        a.region = 0;
        a.q_in = queue[parity];
        a.seg_in = segs[parity];
        a.bitmap_in = bitmap[parity];
        a.bitmap = bitmap[po];
        a.cnt_in = ctl + CTL_BLOCK * parity;
        a.cnt_out = ctl + CTL_BLOCK * po;
        a.q_out = queue[po];
        a.seg_out = segs[po];
        a.work = a.cnt_out + 4;
        const bool dense = cnt[6] > V32 / a.dense_div;
        const uint32_t per = dense ? (uint32_t)kBlock : kMinTile;
        const uint64_t items = (uint64_t)cnt[2] + ((dense ? V32 : cnt[0]) + per - 1) / per;
        const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(items, (uint64_t)sms * 4));
        expand_kernel<kBFS, 1><<<grid, kBlock, 0, s>>>(a);
        build_frontier_kernel<<<fill, kBlock, 0, s>>>(a, bitmap[po], nwords);
        ASC_CUDA(cudaGetLastError());
        ASC_CUDA(cudaMemcpyAsync(cnt, a.cnt_out, sizeof(cnt), cudaMemcpyDeviceToHost, s));
        ASC_CUDA(cudaStreamSynchronize(s));
        parity = po;
    }
    return ASC_OK;
}

// ------------------------------------------------------------- autotuner ----
//
// Picks the engine's tunables for one graph by measurement: the degree above
// which a list is cut into segments, the segment length, the frontier density
// above which a region is walked through its bitmap, and the CTAs per SM of
// the persistent grids. Coordinate descent from the current setting, each
// candidate timed over the given sources (CUDA events, best of two passes).
// Results are cached in a text file keyed by GPU and graph shape
// (ASC_TUNE_CACHE, default $HOME/.cache/ascetic_gb300_tune.txt).
namespace {

std::string tune_key(asc_graph *g, asc_algo algo) {
    cudaDeviceProp prop;
    std::string name = "gpu";
    if (cudaGetDeviceProperties(&prop, g->device) == cudaSuccess) name = prop.name;
    for (auto &c : name)
        if (c == ' ') c = '_';
    char buf[256];
    snprintf(buf, sizeof(buf), "%s:V%llu:E%llu:S%llu:W%u:B%u:C%u:A%d", name.c_str(), (unsigned long long)g->V,
             (unsigned long long)g->E, (unsigned long long)g->static_edges, g->edge_words, g->ebits,
             g->is_csc ? 1 : 0, (int)algo);
    return buf;
}

std::string tune_cache_path() {
    const char *p = getenv("ASC_TUNE_CACHE");
    if (p && *p) return p;
    const char *home = getenv("HOME");
    return std::string(home ? home : "/tmp") + "/.cache/ascetic_gb300_tune.txt";
}

bool tune_cache_lookup(const std::string &key, asc::Tuning *t) {
    FILE *f = fopen(tune_cache_path().c_str(), "r");
    if (!f) return false;
    char line[512], k[256];
    unsigned h, sg, d, c, dl, bu;
    double ms;
    bool found = false;
    // one entry per line: key and the eight fields; lines of another layout are skipped
    while (fgets(line, sizeof(line), f))
        if (sscanf(line, "%255s %u %u %u %u %u %u %lf", k, &h, &sg, &d, &c, &dl, &bu, &ms) == 8 && key == k) {
            t->huge_degree = h;
            t->segment_edges = sg;
            t->dense_div = d;
            t->ctas_per_sm = c;
            t->delta = dl;
            t->bu_div = bu;
            found = true;
        }
    fclose(f);
    return found;
}

void tune_cache_store(const std::string &key, const asc::Tuning &t, double ms) {
    std::string path = tune_cache_path();
    std::string dir = path.substr(0, path.find_last_of('/'));
    if (!dir.empty()) {
        std::string cmd = dir;  // create the cache directory when missing
        mkdir(cmd.c_str(), 0755);
    }
    FILE *f = fopen(path.c_str(), "a");
    if (!f) return;
    fprintf(f, "%s %u %u %u %u %u %u %.4f\n", key.c_str(), t.huge_degree, t.segment_edges, t.dense_div,
            t.ctas_per_sm, t.delta, t.bu_div, ms);
    fclose(f);
}

}  // namespace

namespace asc {

asc_status set_tuning(asc_graph *g, const Tuning &t) {
    if (t.huge_degree < 32 || t.huge_degree > (1u << 20) || t.segment_edges < 256 || t.segment_edges > (1u << 24))
        return fail(ASC_ERR_INVALID, "tuning out of range (huge %u, segment %u)", t.huge_degree, t.segment_edges);
    free_workspace(g);  // segment capacities depend on the thresholds
    g->tuning = t;
    g->has_tuning = true;
    return ASC_OK;
}

}  // namespace asc

extern "C" {

asc_status asc_graph_get_tuning(const asc_graph *g, asc_tuning *t) {
    if (!g || !t) return asc::fail(ASC_ERR_INVALID, "asc_graph_get_tuning: null argument");
    asc::Tuning d;
    if (g->ws) d = g->ws->tune;
    else if (g->has_tuning) d = g->tuning;
    memset(t, 0, sizeof(*t));
    t->huge_degree = d.huge_degree;
    t->segment_edges = d.segment_edges;
    t->dense_div = d.dense_div;
    t->ctas_per_sm = d.ctas_per_sm;
    t->delta = d.delta;
    t->bu_div = d.bu_div;
    return ASC_OK;
}

asc_status asc_graph_set_tuning(asc_graph *g, const asc_tuning *t) {
    if (!g || !t) return asc::fail(ASC_ERR_INVALID, "asc_graph_set_tuning: null argument");
    asc::Tuning x;
    x.huge_degree = t->huge_degree;
    x.segment_edges = t->segment_edges;
    x.dense_div = t->dense_div;
    x.ctas_per_sm = t->ctas_per_sm;
    x.delta = t->delta;
    x.bu_div = t->bu_div;
    return asc::set_tuning(g, x);
}

asc_status asc_graph_tune(asc_graph *g, asc_algo algo, const uint32_t *sources, uint32_t n, uint32_t flags,
                          asc_tuning *best) {
    using namespace asc;
    if (!g || (!sources && algo != ASC_CC && algo != ASC_PR) || (n == 0 && algo != ASC_CC && algo != ASC_PR))
        return fail(ASC_ERR_INVALID, "asc_graph_tune: graph and sources are required");
    if (algo == ASC_PR) return fail(ASC_ERR_UNSUPPORTED, "tuning runs traversals (BFS, SSSP, CC)");
    const std::string key = tune_key(g, algo);
    Tuning cur;
    if (g->ws) cur = g->ws->tune;
    else if (g->has_tuning) cur = g->tuning;
    if (!(flags & ASC_TUNE_NO_CACHE) && tune_cache_lookup(key, &cur)) {
        ASC_TRY(set_tuning(g, cur));
        if (best) ASC_TRY(asc_graph_get_tuning(g, best));
        if (best) best->ms = -1;  // from the cache
        return ASC_OK;
    }
    asc_params p;
    asc_params_default(&p);
    p.flags = ASC_RUN_NO_OUTPUT;
    const uint32_t runs = std::max<uint32_t>(1, std::min<uint32_t>(n, 4));
    auto measure = [&](const Tuning &t, double *ms) -> asc_status {
        ASC_TRY(set_tuning(g, t));
        double bestms = 1e30;
        for (int pass = 0; pass < 2; pass++) {  // first pass warms up (graph build, caches)
            double sum = 0;
            for (uint32_t i = 0; i < runs; i++) {
                asc_stats st;
                ASC_TRY(run_traversal(g, algo, algo == ASC_CC ? 0 : sources[i], p, nullptr, &st));
                sum += st.ms_total;
            }
            bestms = std::min(bestms, sum);
        }
        *ms = bestms;
        return ASC_OK;
    };
    double cur_ms;
    ASC_TRY(measure(cur, &cur_ms));
    const uint32_t huge_c[] = {128, 256, 512, 1024, 4096};
    const uint32_t seg_c[] = {1024, 2048, 4096, 8192};
    const uint32_t div_c[] = {8, 16, 32, 64, 256, 0};
    const uint32_t delta_c[] = {0, 16, 32, 64, 128, 256};
    const uint32_t bu_c[] = {8, 16, 32, 64, 128, 256, 0};
    for (int round = 0; round < 2; round++) {
        if (algo == ASC_BFS && !g->is_csc)
            for (uint32_t b : bu_c) {
                Tuning t = cur;
                t.bu_div = b;
                if (t.bu_div == cur.bu_div) continue;
                double ms;
                ASC_TRY(measure(t, &ms));
                if (ms < cur_ms) { cur = t; cur_ms = ms; }
            }
        if (algo == ASC_SSSP)
            for (uint32_t dl : delta_c) {
                Tuning t = cur;
                t.delta = dl;
                if (t.delta == cur.delta) continue;
                double ms;
                ASC_TRY(measure(t, &ms));
                if (ms < cur_ms) { cur = t; cur_ms = ms; }
            }
        for (uint32_t d : div_c) {
            Tuning t = cur;
            t.dense_div = d;
            if (t.dense_div == cur.dense_div) continue;
            double ms;
            ASC_TRY(measure(t, &ms));
            if (ms < cur_ms) { cur = t; cur_ms = ms; }
        }
        for (uint32_t h : huge_c) {
            Tuning t = cur;
            t.huge_degree = h;
            if (t.huge_degree == cur.huge_degree) continue;
            double ms;
            ASC_TRY(measure(t, &ms));
            if (ms < cur_ms) { cur = t; cur_ms = ms; }
        }
        for (uint32_t sg : seg_c) {
            Tuning t = cur;
            t.segment_edges = sg;
            if (t.segment_edges == cur.segment_edges) continue;
            double ms;
            ASC_TRY(measure(t, &ms));
            if (ms < cur_ms) { cur = t; cur_ms = ms; }
        }
    }
    ASC_TRY(set_tuning(g, cur));
    if (!(flags & ASC_TUNE_NO_CACHE)) tune_cache_store(key, cur, cur_ms / runs);
    if (best) {
        ASC_TRY(asc_graph_get_tuning(g, best));
        best->ms = cur_ms / runs;
    }
    return ASC_OK;
}

}  // extern "C"

extern "C" asc_status asc_graph_fragment_counts(asc_graph *g, uint64_t *out, uint64_t n, uint64_t *n_out, int reset) {
    using namespace asc;
    if (!g) return fail(ASC_ERR_INVALID, "asc_graph_fragment_counts: graph is NULL");
    const uint64_t nf = fragment_count(g);
    if (n_out) *n_out = nf;
    Workspace *ws = g->ws;
    const uint64_t k = std::min(n, nf);
    if (!ws || !ws->frag_counts) {
        if (out) memset(out, 0, 8 * k);
        return ASC_OK;
    }
    if (out && k) {
        ASC_CUDA(cudaMemcpyAsync(out, ws->frag_counts, 8 * k, cudaMemcpyDeviceToHost, g->stream));
    }
    if (reset) ASC_CUDA(cudaMemsetAsync(ws->frag_counts, 0, 8 * std::max<uint64_t>(1, nf), g->stream));
    ASC_CUDA(cudaStreamSynchronize(g->stream));
    return ASC_OK;
}
