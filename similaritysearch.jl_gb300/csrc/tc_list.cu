// tc_list.cu -- tensor-core scan on CTA pairs with the query tile resident and
// append-only candidate lists (tcgen05, cta_group::2).
//
// One scan for every operand form whose 128-query tile fits on chip beside a
// ring of database K-blocks: BF16 and two-piece BF16 rows (64-byte K-blocks,
// tc_bf16.cu), FP8 and wide BF16 rows (128-byte K-blocks, tc_stream.cu), and
// bit sketches as +-1 FP4 rows (Hamming distance = (bits - dot) / 2, exact).
//
// Why lists and a seeded bound.  A search over S splits fills 2 S heaps per
// query, each from scratch: kk (1 + ln(rows / kk)) insertions per heap, and
// while they fill, the slowest of the warps holds its accumulator and with it
// the MMAs (2,048 queries x 1e6 rows x 96 dimensions: 6,400 cycles per
// 128 x 256 tile against 1,940 in allknn, whose order fills the heaps in the
// first tiles).  Long heaps also take the shared memory that the resident
// query tile needs.  Here a first pass over a sample of rows from all over the
// database (SEED, SampleRows) keeps only the smallest distance of each group of columns;
// the kk-th smallest of a query's group minima is a bound with at least kk
// rows at or below it.  The scan then appends what lies at or below that
// bound (about 1.2 kk rows / sample rows per query) to a list in global
// memory: no heap, no sort, no shared memory, and the same kk best keys.
//
// Why pairs.  Each CTA holds its own query tile and half of every database
// K-block; one 256 x 256 MMA reads both.  A K-block byte so feeds 256 query
// rows per SM load: 32 bytes per clock and SM at the full MMA rate instead of
// 64 with one CTA (L2 gives about 35) and 128 for 128 x 128 tiles with both
// operands streamed.
//
// Roles (320 threads per CTA): warp 0 producer, warp 1 TMEM owner and, in the
// even CTA, MMA issuer, warps 2..9 epilogue (two per TMEM lane quarter,
// alternate 32-column chunks of every wide tile, a list each).  Every
// mbarrier wait is bounded (tc_ptx.cuh); both CTAs meet at a cluster barrier
// before TMEM is freed.
#include "common.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"

#include <cuda.h>

#include <algorithm>

namespace ssg {

namespace {

constexpr int TILE = 128;  // query rows per CTA
constexpr int NACC = 2;    // accumulators, of a wide tile's columns each
constexpr int CS = kListSegs;   // epilogue warps per TMEM lane quarter, a list each
constexpr int kThreads = 64 + CS * TILE;
constexpr int kStageBytes = 32 * 1024;  // most of a ring stage
constexpr int kLine = 1024;             // bytes of a tensor-map line
constexpr int kMaxStages = 16;
constexpr size_t kMaxSmem = 227 * 1024;
constexpr size_t kAloneSmem = 120 * 1024;  // all 512 TMEM columns: alone on the SM
constexpr int kCoefBytes = 4 * CS * 2 * (8 / CS) * 128;  // per warp two buffers of a float for each of its columns
constexpr int kTileColumns = 256 / CS;     // columns of a wide tile that one list can take
constexpr int kBufCap = 12;                // raw candidates buffered per lane
constexpr int kBufStride = CS * TILE * 8;  // bytes between a lane's buffer slots
constexpr int kBufBytes = kBufCap * kBufStride;
constexpr int kNextBytes = CS * TILE * 4;  // per lane, the entries beyond which make_room has work

enum { EPI_DOT = LIST_DOT, EPI_SQ = LIST_SQ, EPI_COS = LIST_COS, EPI_AFF = LIST_AFFINE, EPI_HAM = LIST_HAMMING,
       EPI_SCALE = LIST_SCALE };

// EPI_DOT and EPI_HAM rank by the raw product, largest first; the distance is
// made from it only for a candidate.
__host__ __device__ constexpr bool raw_rank(int epi) { return epi == EPI_DOT || epi == EPI_HAM; }
// Floats per database row that the epilogue reads.  Every warp reads them for
// all its columns, as broadcasts of 16 bytes that cost the shared-memory pipe
// as much as 512 bytes of operands: with both factors of AFF for metrics whose
// offset is 0 that was two thirds of what the MMAs' own reads leave (4,096
// queries x 2e6 FP8 rows of 768: 5.42 ms against 5.14 with one).
__host__ __device__ constexpr int coefs(int epi) { return raw_rank(epi) ? 0 : epi == EPI_AFF ? 2 : 1; }

struct KernelArgs {
    ListScan s;
    int kblocks;        // K-blocks per row
    int group;          // K-blocks per ring stage (a divisor of kblocks)
    int stages;         // ring depth
    int64_t n_wide;     // wide tiles of this pass (the sample's in SEED)
    int64_t all_wide;   // of the database
    SampleRows sample;  // SEED: the sampled rows
};

// Keeps the kk smallest of each full list (more than `room` entries): the
// warp takes its lanes' full lists in turn, holds one in registers, finds the
// kk-th key bit by bit and writes the kept keys back.  Returns the calling
// lane's new count and sets *top to its largest kept key.  Lists hold up to
// 32 * PER entries.  A bound seeded from the sample leaves the lists far from
// full unless most of a query's neighbours lie in one split, or its cluster
// lies elsewhere in a locality order; of clusters and duplicates stored side by
// side every query of a tile comes here at once, so registers for lists of 384
// entries have a variant of their own (1,000 queries x 1e5 sketches of two
// words in clusters of 1,000: 348 us, 218 with it and warp_limit).
// BELOW: *top is for a limit just below it.  A lane with more than `next`
// entries, but room for more, then keeps them, and *top is the key `at` of its
// limit; and a distance of +0 is given as -0, which a limit of the next smaller
// float would let through (half a database of zero rows had its lists full
// tile after tile).
template <int PER, bool BELOW>
__device__ __noinline__ int compact_lists(uint64_t *list, int nb, int next, int room, int kk, uint64_t at, uint64_t *top) {
    const int lane = threadIdx.x % 32;
    constexpr uint64_t one = 1ull << 32;
    if (BELOW && nb > next && nb <= room) *top = at >> 32 == 0x80000000u ? at - one : at;
    uint32_t todo = __ballot_sync(0xffffffffu, nb > room);
    while (todo) {
        const int who = __ffs(todo) - 1;
        todo &= todo - 1;
        uint64_t *l = reinterpret_cast<uint64_t *>(
            __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(list), who));
        const int cnt = __shfl_sync(0xffffffffu, nb, who);
        __syncwarp();
        uint64_t key[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) key[i] = i * 32 + lane < cnt ? l[i * 32 + lane] : KEY_EMPTY;
        const uint64_t below = warp_limit<PER>(key, kk);
        int base = 0;
        uint64_t mx = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const bool take = key[i] < below;
            const uint32_t vote = __ballot_sync(0xffffffffu, take);
            const int place = base + __popc(vote & ((1u << lane) - 1u));
            if (take && place < kk) {
                l[place] = key[i];
                mx = key[i] > mx ? key[i] : mx;
            }
            base += __popc(vote);
        }
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t w = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = w > mx ? w : mx;
        }
        __syncwarp();
        if (lane == who) {
            nb = kk;
            *top = BELOW && mx >> 32 == 0x80000000u ? mx - one : mx;
        }
    }
    return nb;
}

// The distance of a ranking value.
template <int EPI>
__device__ __forceinline__ float rank_distance(float x, float bits) {
    return EPI == EPI_DOT ? -x : EPI == EPI_HAM ? (bits - x) * 0.5f : x;
}

// Operand kinds.  Sketches are +-1 in FP4 (e2m1, kind::mxf4 with every scale
// factor 1): half the bytes and MMAs of FP8.  The scale factors take 32 TMEM
// columns, so FP4's accumulators have 240 columns and its database tiles 120
// rows; the others have 256 and 128.
enum { BF16 = 0, FP8 = 1, FP4 = 2 };
__host__ __device__ constexpr int db_rows(int kind) { return kind == FP4 ? 120 : 128; }
constexpr uint32_t kScaleColumns = 480;  // TMEM column of A's scale factors (B's 16 on)

// How a scan orders the database: evenly, as stored; or in a locality order
// (positions with ids, each query tile from its own group on), in one split or
// in several that share what their compactions find.  (Compiled apart: the
// locality order's state cost the batch scans 4 to 12 %, the sharing C2's 5.)
enum { STORED = 0, LOCAL = 1, LOCAL_SHARED = 2 };

// Moves the c raw candidates buffered at shared address buf (slots kBufStride
// apart: ranking value, position) to the lane's list, as keys; those beyond
// the largest key a compaction kept are left out.  All 32 lanes call it, with
// scalars alone and few registers of its own, so the call saves nothing.
template <int EPI, int ORDER>
__device__ __noinline__ int drain_raw(uint64_t *list, uint32_t buf, int c, int nb, float bits, uint64_t top,
                                      const uint32_t *perm) {
    const int cmax = __reduce_max_sync(0xffffffffu, c);
    for (int i = 0; i < cmax; ++i) {
        if (i < c) {
            float v;
            uint32_t pos;
            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=f"(v), "=r"(pos) : "r"(buf + i * kBufStride) : "memory");
            const uint64_t key = make_key(rank_distance<EPI>(v, bits), ORDER != STORED ? perm[pos] : pos);
            if (ORDER == STORED || key <= top) list[nb++] = key;
        }
    }
    return nb;
}

// One query row's candidates (one lane).
template <int EPI, int ORDER>
struct RowList {
    uint64_t *list;
    uint32_t buf;      // shared address of this lane's raw buffer
    int nb, nbuf, cap, kk;
    uint64_t top;      // the largest key kept by the last compaction
    const uint32_t *perm;
    int64_t n;
    bool valid;
    float lim_v;       // a candidate's ranking value: product >= lim_v (raw_rank) or distance <= lim_v
    float bits;        // EPI_HAM: bits per sketch
    float gamma;       // EPI_AFF, EPI_SCALE: the query's scale

    // the limit for a bound t on the distance; a row that is no query's lets nothing through
    __device__ __forceinline__ void set(float t) {
        if (!valid) t = -INFINITY;
        lim_v = EPI == EPI_HAM ? bits - 2.0f * t : EPI == EPI_DOT ? -t : t;
    }
    // ranking values of a chunk's 32 columns: products (raw_rank) or distances
    // (al, be: the columns' coefficients in shared memory)
    __device__ __forceinline__ void values(const uint32_t (&r)[32], const float4 *al, const float4 *be,
                                           float (&dv)[32]) const {
        if constexpr (raw_rank(EPI)) {
#pragma unroll
            for (int j = 0; j < 32; ++j) dv[j] = __uint_as_float(r[j]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 a = al[j];
                const float v0 = __uint_as_float(r[4 * j]), v1 = __uint_as_float(r[4 * j + 1]);
                const float v2 = __uint_as_float(r[4 * j + 2]), v3 = __uint_as_float(r[4 * j + 3]);
                if constexpr (EPI == EPI_SQ) {
                    dv[4 * j] = fmaf(-2.0f, v0, a.x);
                    dv[4 * j + 1] = fmaf(-2.0f, v1, a.y);
                    dv[4 * j + 2] = fmaf(-2.0f, v2, a.z);
                    dv[4 * j + 3] = fmaf(-2.0f, v3, a.w);
                } else if constexpr (EPI == EPI_COS) {
                    dv[4 * j] = -v0 * a.x;
                    dv[4 * j + 1] = -v1 * a.y;
                    dv[4 * j + 2] = -v2 * a.z;
                    dv[4 * j + 3] = -v3 * a.w;
                } else {
                    const float4 b = EPI == EPI_AFF ? be[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    dv[4 * j] = fmaf(v0 * gamma, a.x, b.x);
                    dv[4 * j + 1] = fmaf(v1 * gamma, a.y, b.y);
                    dv[4 * j + 2] = fmaf(v2 * gamma, a.z, b.z);
                    dv[4 * j + 3] = fmaf(v3 * gamma, a.w, b.w);
                }
            }
        }
    }
    __device__ __forceinline__ static float best8(const float *v) { return raw_rank(EPI) ? fmax8(v) : fmin8(v); }
    __device__ __forceinline__ static float best(float a, float b) { return raw_rank(EPI) ? fmaxf(a, b) : fminf(a, b); }
    __device__ __forceinline__ bool passes(float x) const { return raw_rank(EPI) ? x >= lim_v : x <= lim_v; }

    // The best ranking value at each of P places of a chunk's atoms of 8 rows
    // (columns p, p + P, ...), with those before it.
    // (cols: the chunk's columns that are the tile's)
    template <int P>
    __device__ __forceinline__ void places(const uint32_t (&r)[32], int cols, const float4 *al, const float4 *be,
                                           float (&g)[P]) const {
        float dv[32];
        values(r, al, be, dv);
#pragma unroll
        for (int j = 0; j < 32; j += 2 * P) {
            if (j >= 16 && cols != 32) break;
#pragma unroll
            for (int i = 0; i < P; ++i)
                g[i] = raw_rank(EPI) ? fmax3(g[i], dv[j + i], dv[j + P + i]) : fmin3(g[i], dv[j + i], dv[j + P + i]);
        }
    }
    template <int P>
    __device__ __forceinline__ static void no_places(float (&g)[P]) {
#pragma unroll
        for (int i = 0; i < P; ++i) g[i] = raw_rank(EPI) ? -INFINITY : INFINITY;
    }
    __device__ __forceinline__ void drain() {
        nb = drain_raw<EPI, ORDER>(list, buf, nbuf, nb, bits, ORDER != STORED ? top : KEY_EMPTY, ORDER != STORED ? perm : nullptr);
        nbuf = 0;
    }
    // Between tiles (nothing of an accumulator in registers): makes room for
    // another tile's columns in every list of the warp.
    // Where rows come as stored a list is looked at once before, when it has kk
    // entries: equal rows would fill it first (2,563 queries x 29,191 equal
    // sketches 444 -> 184 us; allknn of 51,601 BF16 rows of 11, half of them
    // zeros, 15.7 -> 1.2 ms).  next_at is the shared address of the lane's
    // threshold: as a register it cost a scan of sketches 9 %.
    __device__ __forceinline__ bool make_room(uint32_t next_at) {
        const int room = cap - kTileColumns - kBufCap;
        int next = room;
        if (ORDER == STORED) {
            // (most lists never have kk: the load waits 1 % of a tile)
            if (!__any_sync(0xffffffffu, nb >= kk)) return false;
            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(next) : "r"(next_at));
        }
        if (!__any_sync(0xffffffffu, nb > next)) return false;
        drain();
        if (ORDER == STORED && nb > next) asm volatile("st.shared.b32 [%0], %1;" ::"r"(next_at), "r"(room) : "memory");
        uint64_t t = 0;
        const uint64_t at = ORDER == STORED ? make_key(limit(), 0) : 0;
        nb = cap <= 384 ? compact_lists<12, ORDER == STORED>(list, nb, next, room, kk, at, &t)
                        : compact_lists<kListMaxCap / 32, ORDER == STORED>(list, nb, next, room, kk, at, &t);
        if (t) {
            // kk keys up to t are kept, or there are kk within the limit.  Ids
            // only grow from here where rows come as stored: an equal distance
            // no longer counts.  Positions of a locality order have any ids:
            // the drain compares the keys.
            if (ORDER != STORED) top = t;
            const float d = key_dist(t);
            const float e = ORDER != STORED ? d : EPI == EPI_HAM ? d - 0.5f : ordered_to_float(uint32_t(t >> 32) - 1u);
            const float v = EPI == EPI_HAM ? bits - 2.0f * e : EPI == EPI_DOT ? -e : e;
            lim_v = raw_rank(EPI) ? fmaxf(lim_v, v) : fminf(lim_v, v);
        }
        return true;
    }
    // The limit as a bound on the distance, and back: what a compaction found
    // holds for every list of the query.
    __device__ __forceinline__ float limit() const {
        return EPI == EPI_HAM ? (bits - lim_v) * 0.5f : EPI == EPI_DOT ? -lim_v : lim_v;
    }
    __device__ __forceinline__ void publish(uint32_t *bound) const {
        if (valid && top != KEY_EMPTY) bound_lower(bound, limit());
    }
    __device__ __forceinline__ void refresh(const uint32_t *bound) {
        if (!valid) return;
        const float t = bound_read(bound);
        const float v = EPI == EPI_HAM ? bits - 2.0f * t : EPI == EPI_DOT ? -t : t;
        lim_v = raw_rank(EPI) ? fmaxf(lim_v, v) : fminf(lim_v, v);
    }
    // Candidates of a chunk: a vote on the chunk and on each group of 8
    // columns, then branch-free raw appends (the slot is always written, the
    // count only advances for a candidate) to a buffer that is drained when a
    // lane has more than kBufCap - 8.  Anything dearer per group held up the
    // MMAs: 2,048 queries x 1e6 rows x 96 dimensions took 691 us with the
    // keys appended at the sites, 497 through a function (its calls spilled
    // the accumulator's registers), 356 so.
    __device__ __forceinline__ void chunk(const uint32_t (&r)[32], int64_t id0, int cols, const float4 *al,
                                          const float4 *be) {
        float dv[32], g[4];
        values(r, al, be, dv);
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] = best8(dv + 8 * i);
        if (!__any_sync(0xffffffffu, passes(best(best(g[0], g[1]), best(g[2], g[3]))))) return;
        const int lim = !valid ? 0 : id0 + cols <= n ? cols : int(n - id0);  // columns that are rows
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!__any_sync(0xffffffffu, passes(g[i]))) continue;
#pragma unroll
            for (int j = 8 * i; j < 8 * i + 8; ++j) {
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(buf + nbuf * kBufStride), "f"(dv[j]),
                             "r"(uint32_t(id0) + uint32_t(j))
                             : "memory");
                nbuf += (passes(dv[j]) && j < lim) ? 1 : 0;
            }
            if (__any_sync(0xffffffffu, nbuf > kBufCap - 8)) drain();
        }
    }
};

// QSTREAM: the query tile does not fit on chip; its K-blocks come through the
// ring beside the database's (64 bytes per clock and SM at the full MMA rate,
// half of what 128 x 128 tiles take).
template <int SWB, int KIND, int EPI, bool SEED, int ORDER, bool QSTREAM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    tc_list_kernel(KernelArgs ka, const __grid_constant__ CUtensorMap dmap, const __grid_constant__ CUtensorMap qmap) {
    constexpr int HROWS = db_rows(KIND);  // database rows per tile
    constexpr int WIDE = 2 * HROWS;       // and per MMA: a tile of each CTA
    constexpr int KBLK = TILE * SWB;      // bytes of a K-block of a query tile
    constexpr int DBLK = HROWS * SWB;     // and of a database tile
    constexpr int KSTEPS = SWB / 32;   // MMAs per K-block (32 bytes of K each)
    const ListScan &a = ka.s;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int kblocks = ka.kblocks, stages = ka.stages, group = ka.group;
    const int groups_per_tile = kblocks / group;
    const size_t tile_bytes = size_t(kblocks) * KBLK;
    const uint32_t part_bytes = uint32_t(group) * DBLK;
    const uint32_t stage_bytes = (QSTREAM ? 2 : 1) * part_bytes;  // (QSTREAM: KBLK = DBLK)
    uint8_t *sA = smem;
    uint8_t *sB = sA + (QSTREAM ? 0 : tile_bytes);  // stages: database part, then the query part
    // per epilogue warp, two buffers of its 64 columns' coefficients
    float4 *coef = reinterpret_cast<float4 *>(sB + size_t(stages) * stage_bytes);
    uint64_t *bufs = reinterpret_cast<uint64_t *>(coef + coefs(EPI) * kCoefBytes / 16);  // raw candidates
    uint64_t *bars = bufs + (SEED ? 0 : (kBufBytes + kNextBytes) / 8);
    uint64_t *a_full = bars;                  // this CTA's query tile landed
    uint64_t *pa_full = a_full + 1;           // (even CTA) the odd CTA's query tile landed
    uint64_t *full = pa_full + 1;             // (even CTA) both halves of stage s landed
    uint64_t *empty = full + kMaxStages;      // the MMAs of stage s are done
    uint64_t *acc_full = empty + kMaxStages;  // accumulator b holds a finished tile
    uint64_t *acc_empty = acc_full + NACC;    // (even CTA) the epilogue warps of both CTAs released b
    uint64_t *mma_done = acc_empty + NACC;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t rank = tc::cluster_ctarank();  // 0: the even CTA (issues the MMAs)
    const uint32_t peer = rank ^ 1u;
    const int64_t qx = blockIdx.x;                // this CTA's query tile
    const int64_t qpair = qx - int64_t(rank);
    // epilogue warps of the pair whose lane quarter holds a query
    int live = 0;
    for (int w = 0; w < 8; ++w)
        if (qpair * TILE + w * 32 < a.m) live += CS;

    if (threadIdx.x == 0) {
        tc::mbar_init(a_full, 1);
        tc::mbar_init(pa_full, 1);
        for (int s = 0; s < stages; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < NACC; ++b) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], live);
        }
        tc::mbar_init(mma_done, 1);
        tc::fence_mbarrier_init();
    }
    if (warp == 1) tc::tmem_alloc_pair<512>(tmem_slot);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // behind this block's allocation: no later kernel's block can take the
    // TMEM first and then wait for this one.  (Not the scan's: finalize blocks
    // held on its SMs cost 45 us of 2,680.)
    if (SEED) griddep_launch();
    if constexpr (KIND == FP4) {
        // every scale factor is 1 (UE8M0 127), so their layout does not matter
        if (warp >= 2 && warp < 6) {
            tc::tmem_st_32x32b_x32(tmem_base + (uint32_t(warp % 4 * 32) << 16) + kScaleColumns, 0x7f7f7f7fu);
            tc::tmem_wait_st();
        }
        tc::tc_fence_before();
        __syncthreads();
    }
    tc::cluster_sync();  // both CTAs' barriers (and scale factors) exist before any cross-CTA arrive
    griddep_wait();
    tc::tc_fence_after();

    // this split's wide tiles (places in the sample when SEED)
    const int64_t split_w = (ka.n_wide + a.splits - 1) / a.splits;
    const int64_t w_lo = int64_t(blockIdx.y) * split_w;
    const int64_t w_hi = w_lo + split_w < ka.n_wide ? w_lo + split_w : ka.n_wide;
    const int W = w_hi > w_lo ? int(w_hi - w_lo) : 0;
    // the u-th wide tile: of the whole scan, from the locality rotation on; in
    // SEED of the tiles around the rotation (the sample of a stored order is
    // put together from atoms)
    int64_t first = ORDER != STORED ? int64_t(a.rot[qpair]) / 2 : 0;
    if (SEED && ORDER != STORED) first = first >= a.samples / 2 ? first - a.samples / 2 : first - a.samples / 2 + ka.all_wide;
    constexpr bool SPREAD = SEED && ORDER == STORED;  // sampled rows from all over the database
    constexpr int ATOMS = HROWS / 8;
    auto wide_tile = [&](int u) {
        if (ORDER == STORED) return w_lo + u;
        const int64_t p = w_lo + u + first;
        return p >= ka.all_wide ? p - ka.all_wide : p;
    };

    if (warp == 0) {
        if (lane == 0) {
            // producer: this CTA's query tile, then its tile's part of
            // every K-block group; both halves of a stage complete on the
            // even CTA's full[s]
            if constexpr (!QSTREAM) {
                tc::mbar_arrive_expect_tx(a_full, uint32_t(tile_bytes));
                for (int kb = 0; kb < kblocks; ++kb)
                    tc::bulk_g2s(sA + size_t(kb) * KBLK, a.qt + size_t(qx) * tile_bytes + size_t(kb) * KBLK, KBLK,
                                 a_full);
            }
            const uint32_t full0 = tc::mapa_shared(tc::smem_u32(full), 0);
            int s = 0, issued = 0;
            uint32_t ph = 1;
            bool ok = true;
            int unit = SPREAD ? sample_first(ka.sample, w_lo) : 0;
            for (int u = 0; ok && u < W; ++u) {
                int line = (int(wide_tile(u)) * 2 + int(rank)) * kblocks * (DBLK / kLine);
                int64_t tile0 = 0;
                int atom = 0;
                if (SPREAD) {
                    sample_unit(ka.sample, ATOMS, unit + int(rank) * ka.sample.samples, &tile0, &atom);
                    unit = sample_next(ka.sample, unit);
                }
                int qline = int(qx) * kblocks * (KBLK / kLine);
                for (int g = 0; g < groups_per_tile; ++g, line += group * (DBLK / kLine)) {
                    if (!tc::mbar_wait(&empty[s], ph, a.err, 21)) { ok = false; break; }
                    if (rank == 0) tc::mbar_arrive_expect_tx(&full[s], 2 * stage_bytes);
                    uint8_t *dst = sB + size_t(s) * stage_bytes;
                    if constexpr (SPREAD) {
                        for (int kb = 0; kb < group; ++kb)
                            tc::tma_load_5d_pair(dst + kb * DBLK, &dmap, 0, atom, g * group + kb, int(tile0), 0,
                                                 full0 + uint32_t(s * 8));
                    } else {
                        tc::tma_load_2d_pair(dst, &dmap, 0, line, full0 + uint32_t(s * 8));
                    }
                    if constexpr (QSTREAM) {
                        tc::tma_load_2d_pair(dst + part_bytes, &qmap, 0, qline, full0 + uint32_t(s * 8));
                        qline += group * (KBLK / kLine);
                    }
                    issued = issued < stages ? issued + 1 : stages;
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
            }
            // wait (bounded) until every copy of this pair has landed (the
            // even CTA's barriers count both halves; the final cluster
            // barrier keeps the odd CTA alive until then)
            if (!QSTREAM) tc::mbar_wait(a_full, 0, a.err, 22);
            if (rank == 0) {
                // the last `issued` stages, newest first: a stage's landing
                // phase is the opposite of the one its emptiness was waited for
                for (int i = 0; i < issued; ++i) {
                    if (--s < 0) { s = stages - 1; ph ^= 1; }
                    tc::mbar_wait(&full[s], ph ^ 1, a.err, 22);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 1) {
            // the odd CTA tells the even CTA that its query tile landed
            if (!QSTREAM && tc::mbar_wait(a_full, 0, a.err, 28)) tc::mbar_arrive_cluster(tc::mapa_shared(tc::smem_u32(pa_full), peer));
        } else if (lane == 0) {
            // the even CTA issues the pair's MMAs
            constexpr uint32_t idesc = KIND == FP4   ? tc::idesc_mxf4_f32(2 * TILE, WIDE)
                                       : KIND == FP8 ? tc::idesc_e4m3_f32(2 * TILE, WIDE)
                                                     : tc::idesc_bf16_f32(2 * TILE, WIDE);
            bool ok = QSTREAM || (tc::mbar_wait(a_full, 0, a.err, 23) && tc::mbar_wait(pa_full, 0, a.err, 23));
            // descriptors address 16-byte units
            const uint64_t a_desc = tc::smem_desc(tc::smem_u32(sA), SWB);
            const uint64_t b_desc = tc::smem_desc(tc::smem_u32(sB), SWB);
            int s = 0, b = 0;
            uint32_t ph = 0, aph = 1;
            for (int u = 0; ok && u < W; ++u) {
                if (!tc::mbar_wait(&acc_empty[b], aph, a.err, 25)) break;
                const uint32_t d_tmem = tmem_base + uint32_t(b * WIDE);
                uint64_t ad = a_desc;
                uint32_t acc = 0;
                for (int g = 0; g < groups_per_tile; ++g) {
                    if (!tc::mbar_wait(&full[s], ph, a.err, 24)) { ok = false; break; }
                    tc::tc_fence_after();
                    uint64_t bd = b_desc + uint64_t((uint32_t(s) * stage_bytes) >> 4);
                    if (QSTREAM) ad = bd + uint64_t(part_bytes >> 4);
                    for (int kb = 0; kb < group; ++kb) {
#pragma unroll
                        for (int k = 0; k < KSTEPS; ++k) {
                            if (KIND == FP4)
                                tc::mma_mxf4_pair(d_tmem, ad + 2 * k, bd + 2 * k, idesc, tmem_base + kScaleColumns,
                                                  tmem_base + kScaleColumns + 16, k ? 1u : acc);
                            else if (KIND == FP8) tc::mma_f8_pair(d_tmem, ad + 2 * k, bd + 2 * k, idesc, k ? 1u : acc);
                            else tc::mma_f16_pair(d_tmem, ad + 2 * k, bd + 2 * k, idesc, k ? 1u : acc);
                        }
                        acc = 1;
                        ad += KBLK >> 4;
                        bd += DBLK >> 4;
                    }
                    tc::mma_commit_both(&empty[s]);
                    if (++s == stages) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
                tc::mma_commit_both(&acc_full[b]);
                if (++b == NACC) { b = 0; aph ^= 1; }
            }
            tc::mma_commit_pair(tc::smem_u32(mma_done));
            tc::mbar_wait(mma_done, 0, a.err, 26);
        }
        __syncwarp();
    } else {
        const int cs = (warp - 2) / 4;
        const int quarter = warp % 4;
        const int64_t query = qx * TILE + quarter * 32 + lane;
        const uint32_t release0 = tc::mapa_shared(tc::smem_u32(acc_empty), 0);
        const int seg = int(blockIdx.y) * CS + cs, segs = a.splits * CS;
        RowList<EPI, ORDER> T;
        T.valid = query < a.m;
        T.list = SEED ? nullptr : a.lists + (size_t(T.valid ? query : 0) * segs + seg) * a.cap;
        T.nb = 0;
        T.nbuf = 0;
        T.buf = tc::smem_u32(bufs) + uint32_t((warp - 2) * 32 + lane) * 8;
        T.cap = a.cap;
        T.kk = a.kk;
        T.n = a.n;
        T.top = KEY_EMPTY;
        T.perm = a.perm;
        T.bits = a.bits;
        T.gamma = ((EPI == EPI_AFF || EPI == EPI_SCALE) && a.gamma && T.valid) ? a.gamma[query] : 1.0f;
        // the lane's word behind the buffers, half of its slots' stride
        const uint32_t next_at = (T.buf >> 1) + (tc::smem_u32(bufs) + kBufBytes - (tc::smem_u32(bufs) >> 1));
        if (!SEED && ORDER == STORED) asm volatile("st.shared.b32 [%0], %1;" ::"r"(next_at), "r"(a.kk - 1) : "memory");
        T.set((!SEED && T.valid) ? bound_read(a.bound + query) : INFINITY);
        const bool warp_live = qx * TILE + quarter * 32 < a.m;
        // this warp's columns of a wide tile: the 32-column chunks cs, cs + CS, ...;
        // their coefficients are copied a tile ahead
        constexpr int CH = 8 / CS;
        float4 *mine = coef + (warp - 2) * coefs(EPI) * CH * 16;
        int unit = SPREAD ? sample_first(ka.sample, w_lo) : 0;
        auto fetch = [&](int u, int buf) {
            if constexpr (!raw_rank(EPI)) {
                constexpr int PER = CH * 8;  // 16-byte pieces of alpha, and of beta
                for (int p = lane; p < coefs(EPI) * PER; p += 32) {
                    const int col = (cs + CS * (p % PER / 8)) * 32 + (p % 8) * 4;
                    int64_t row = wide_tile(u) * WIDE + col;
                    if constexpr (SPREAD) {
                        int64_t tile0;
                        int atom;
                        sample_unit(ka.sample, ATOMS, unit + col / HROWS * ka.sample.samples, &tile0, &atom);
                        row = sample_row(ka.sample, HROWS, tile0, atom, col % HROWS);
                    }
                    const float *src = (p < PER ? a.alpha : a.beta) + row;
                    const uint32_t d = tc::smem_u32(mine + buf * coefs(EPI) * PER + p);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
                }
                if (SPREAD) unit = sample_next(ka.sample, unit);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
        };
        if (warp_live && W > 0) fetch(0, 0);
        float place[4];  // SEED: the best ranking value at each second place of the sampled atoms
        T.no_places(place);
        int b = 0;
        uint32_t ph = 0;
        for (int u = 0; warp_live && u < W; ++u) {
            int ok = 1;
            if (lane == 0) ok = tc::mbar_wait(&acc_full[b], ph, a.err, 27) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            tc::tc_fence_after();
            // all four chunks in flight together where their products are
            // the ranking values, and the accumulator back before any is
            // looked at; two rounds of two where the distances take registers
            // too.  (Sixteen warps with two chunks each release as early but
            // crowd the MMA thread: 10,000 queries x 2e6 sketches, then in FP8,
            // 11.8 ms against 10.4.)
            constexpr int LDC = raw_rank(EPI) ? 4 : 2;
            const uint32_t tbase = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(b * WIDE + cs * 32);
            const int64_t row0 = (SPREAD ? 0 : wide_tile(u) * WIDE) + cs * 32;  // (all sampled places are rows)
            const float4 *al = mine + (u & 1) * (coefs(EPI) * CH * 8);  // alpha, then beta
            uint32_t r[LDC][32];
#pragma unroll
            for (int round = 0; round < CH / LDC; ++round) {
                __syncwarp();
#pragma unroll
                for (int c = 0; c < LDC; ++c) {
                    const uint32_t from = tbase + uint32_t((round * LDC + c) * CS * 32);
                    // (FP4's wide tile ends after 16 columns of the last chunk)
                    if (KIND == FP4 && round * LDC + c == CH - 1 && cs == CS - 1) tc::tmem_ld_32x32b_x16_async(from, r[c]);
                    else tc::tmem_ld_32x32b_x32_async(from, r[c]);
                }
                if constexpr (!raw_rank(EPI)) {
                    if (round == 0) {
                        if (u + 1 < W) fetch(u + 1, (u + 1) & 1);
                        else asm volatile("cp.async.commit_group;" ::: "memory");
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                    }
                }
                tc::tmem_wait_ld();
                if (round == CH / LDC - 1) tc::tc_fence_before();
                __syncwarp();
                if (round == CH / LDC - 1 && lane == 0) {
                    if (rank == 0) tc::mbar_arrive(&acc_empty[b]);
                    else tc::mbar_arrive_cluster_relaxed(release0 + uint32_t(b * 8));
                }
#pragma unroll
                for (int c = 0; c < LDC; ++c) {
                    const int ch = round * LDC + c;
                    const int col0 = (cs + ch * CS) * 32;
                    const int cols = WIDE == 256 || col0 + 32 <= WIDE ? 32 : WIDE - col0;
                    if constexpr (SEED) {
                        if (SPREAD && a.per_tile != 64) {
                            T.places(r[c], cols, al + ch * 8, al + CH * 8 + ch * 8, place);
                        } else if (T.valid) {
                            float g[8];
                            T.no_places(g);
                            T.places(r[c], cols, al + ch * 8, al + CH * 8 + ch * 8, g);
                            // (a locality order's last tile has columns that are no rows)
                            const bool rows = SPREAD || row0 + ch * CS * 32 + cols <= a.n;
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                g[i] = rows ? fminf(rank_distance<EPI>(g[i], a.bits), INFINITY) : INFINITY;
                            float4 *to = reinterpret_cast<float4 *>(a.minima + size_t(query) * a.groups + (w_lo + u) * 64 +
                                                                    (cs * CH + ch) * 8);
                            to[0] = make_float4(g[0], g[1], g[2], g[3]);
                            to[1] = make_float4(g[4], g[5], g[6], g[7]);
                        }
                    } else T.chunk(r[c], row0 + ch * CS * 32, cols, al + ch * 8, al + CH * 8 + ch * 8);
                }
            }
            if (++b == NACC) { b = 0; ph ^= 1; }
            if constexpr (SPREAD) {
                // a warp's minima go to its wide tile's four slots, or those of
                // four wide tiles to a slot of each (fewer at a split's end
                // join places)
                const int in = a.per_tile == 8 ? 1 : (u & 3) + 1;
                if (a.per_tile != 64 && (a.per_tile == 8 || in == 4 || u + 1 == W)) {
                    if (T.valid) {
                        float *to = a.minima + size_t(query) * a.groups + (w_lo + u + 1 - in) * a.per_tile;
#pragma unroll
                        for (int i = 0; i < 4; ++i) place[i] = fminf(rank_distance<EPI>(place[i], a.bits), INFINITY);  // (a NaN: +inf)
                        if (a.per_tile == 8) {
                            *reinterpret_cast<float4 *>(to + cs * 4) = make_float4(place[0], place[1], place[2], place[3]);
                        } else {
                            if (in == 1) place[0] = fminf(place[0], place[1]);
                            if (in <= 2) place[0] = fminf(place[0], place[2]);
                            if (in == 2) place[1] = fminf(place[1], place[3]);
                            else if (in < 4) place[0] = fminf(place[0], place[3]);
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                if (t < in) to[t * CS + cs] = place[t];
                        }
                    }
                    T.no_places(place);
                }
            }
            if constexpr (!SEED) {
                const bool tighter = T.make_room(next_at);
                if (ORDER == LOCAL_SHARED) {
                    if (tighter) T.publish(a.bound + query);
                    else if ((u & 15) == 15) T.refresh(a.bound + query);
                }
            }
            if constexpr (!raw_rank(EPI)) __syncwarp();  // the buffer is refilled a tile later
        }
        if (!raw_rank(EPI)) asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (!SEED && warp_live) T.drain();
        if (!SEED && T.valid) a.counts[size_t(query) * segs + seg] = T.nb;
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::cluster_sync();  // the even CTA's MMAs are done with both CTAs' shared memory
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc_pair<512>(tmem_base);
    }
}

// bound[q] = the kk-th smallest of the query's group minima (all ones, no
// bound, when they are not that many): each is the distance of another row.
// A warp per query; groups beyond 32 * NV are joined (their minimum is still
// a row's distance), the kk-th value is found bit by bit from registers.
template <int NV>
__global__ void __launch_bounds__(128) seed_bound_kernel(const float *minima, int64_t m, int groups, int kk,
                                                         uint32_t *bound) {
    griddep_launch();
    griddep_wait();
    const int64_t q = int64_t(blockIdx.x) * 4 + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (q >= m) return;
    const float *g = minima + size_t(q) * groups;
    float f[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) f[i] = i * 32 + lane < groups ? __ldcg(g + i * 32 + lane) : INFINITY;
    for (int at = NV * 32 + lane; at < groups; at += NV * 32) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (at + i * 32 < groups) f[i] = fminf(f[i], __ldcg(g + at + i * 32));
    }
    uint32_t v[NV], lo = 0xffffffffu, hi = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        v[i] = float_to_ordered(f[i]);
        lo = min(lo, v[i]);
        hi = max(hi, v[i]);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    // the bits above the highest one in which two minima differ are common;
    // with exactly kk minima below t any value from the kk-th to t - 1 will do
    const int top = 31 - __clz((lo ^ hi) | 1u);
    uint32_t p = top >= 31 ? 0u : (lo >> (top + 1)) << (top + 1);
    for (int b = top; b >= 0; --b) {
        const uint32_t t = p | (1u << b);
        int c = 0;
#pragma unroll
        for (int i = 0; i < NV; ++i) c += v[i] < t;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c == kk) { p = t - 1; break; }
        if (c < kk) p = t;
    }
    if (lane == 0) bound[q] = kk <= groups ? p : 0xffffffffu;
}

// Sketches -> +-1 FP4 (e2m1) tiles of tile_rows rows in the 128-byte K-block
// layout: bit 0 is +1 (2), bit 1 is -1 (10), words past the sketch and rows past
// the end are zeros.  Thread = 32 bits = one 16-byte chunk.
__global__ void sketch_tile_kernel(const uint64_t *__restrict__ x, int64_t rows, int words, int kblocks, int tile_rows,
                                   int64_t tiles, uint8_t *__restrict__ out) {
    griddep_launch();
    const int chunks = kblocks * 8;  // 32-bit chunks per padded row
    const int64_t total = tiles * tile_rows * chunks;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x) {
        const int ch = int(i % chunks);
        const int64_t row = i / chunks;
        uint32_t w[4] = {0, 0, 0, 0};
        if (row < rows && ch < words * 2) {
            const uint32_t bits = uint32_t(x[row * words + ch / 2] >> ((ch % 2) * 32));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // eight bits spread to the nibbles' sign bits
                uint32_t b = (bits >> (8 * k)) & 0xffu;
                b = (b | (b << 12)) & 0x000f000fu;
                b = (b | (b << 6)) & 0x03030303u;
                b = (b | (b << 3)) & 0x11111111u;
                w[k] = (b << 3) | 0x22222222u;
            }
        }
        const int64_t tile = row / tile_rows;
        const uint32_t off = tc::swizzled_offset(uint32_t(row % tile_rows), uint32_t((ch % 8) * 16), 128);
        uint8_t *dst = out + (size_t(tile) * kblocks + ch / 8) * (tile_rows * 128) + off;
        *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// The database tiles as lines of 1 KB (128 eight-byte elements; the bytes are
// already swizzled, so a box is copied verbatim): a box is one tile's part of
// a ring stage, a whole row's K-blocks where they fit.
// (rank 5: the seed's sample, an atom of 8 rows at a time)
cudaError_t encode_map(const uint8_t *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                       const cuuint32_t *box, CUtensorMap *map) {
    using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    if (reinterpret_cast<uintptr_t>(base) % 16 != 0) return cudaErrorInvalidValue;
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, cuuint32_t(rank), const_cast<uint8_t *>(base), dims,
                              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t line_map(const uint8_t *base, int64_t bytes, int64_t box_bytes, CUtensorMap *map) {
    const cuuint64_t dims[2] = {cuuint64_t(kLine / 8), cuuint64_t(bytes / kLine)};
    const cuuint64_t strides[1] = {cuuint64_t(kLine)};
    const cuuint32_t box[2] = {cuuint32_t(kLine / 8), cuuint32_t(box_bytes / kLine)};
    return encode_map(base, 2, dims, strides, box, map);
}

// The sample: a box is a K-block of one unit (SampleRows), an atom of 8 rows
// from each of its tiles; coordinates (0, line of atoms, K-block, first tile, 0).
cudaError_t sample_map(const uint8_t *base, int tile_rows, int swb, int kblocks, int64_t q, CUtensorMap *map) {
    const cuuint64_t atoms = cuuint64_t(tile_rows / 8), atom = cuuint64_t(8 * swb), block = atoms * atom;
    const cuuint64_t dims[5] = {atom / 8, atoms, cuuint64_t(kblocks), cuuint64_t(q), atoms};
    const cuuint64_t strides[4] = {atom, block, cuuint64_t(kblocks) * block, cuuint64_t(q) * cuuint64_t(kblocks) * block};
    const cuuint32_t box[5] = {cuuint32_t(atom / 8), 1, 1, 1, cuuint32_t(atoms)};
    return encode_map(base, 5, dims, strides, box, map);
}

size_t list_smem(int query_bytes, int stage_bytes, int stages, int epi) {
    return 1024 + size_t(query_bytes) + size_t(stages) * stage_bytes + coefs(epi) * kCoefBytes + kBufBytes + kNextBytes +
           (2 + 2 * kMaxStages + 2 * NACC + 1) * 8 + 16;
}

// The ring: K-blocks per stage (a divisor of the row's) and stages, beside a
// resident query tile or with its K-blocks in the stages.  Every stage costs
// the MMA thread a wait and a commit, so the largest stages of which three
// fit, up to 32 KB (2,048 queries x 1e6 rows of 96 dimensions: the seed 51 us
// with a K-block per stage, 35 with the row's three).  stages = 0: not even
// four K-blocks fit.
struct Ring {
    int group, stages;
    bool qstream;
    size_t smem;
};
Ring list_ring(int row_bytes, int swb, int epi) {
    const int kblocks = row_bytes / swb;
    const int rows = db_rows(epi == EPI_HAM ? FP4 : BF16);
    for (int qstream = 0; qstream < 2; ++qstream) {
        const int query_bytes = qstream ? 0 : TILE * row_bytes, parts = qstream ? 2 : 1;
        for (int g = std::min(kblocks, kStageBytes / (TILE * swb)); g >= 1; --g) {
            if (kblocks % g) continue;
            const int stage = parts * g * rows * swb;
            int st = kMaxStages;
            while (st > 0 && list_smem(query_bytes, stage, st, epi) > kMaxSmem) --st;
            if (st >= 3 && st * g >= 4) return {g, st, qstream != 0, list_smem(query_bytes, stage, st, epi)};
        }
    }
    return {1, 0, false, 0};
}

template <int SWB, int KIND, int EPI, bool SEED, int ORDER, bool QSTREAM>
cudaError_t launch_list_q(const ListScan &s, const Ring &ring, cudaStream_t st) {
    KernelArgs ka;
    ka.s = s;
    ka.kblocks = s.row_bytes / SWB;
    ka.group = ring.group;
    ka.stages = ring.stages;
    constexpr int rows = db_rows(KIND);
    ka.all_wide = (s.n + 2 * rows - 1) / (2 * rows);
    ka.n_wide = SEED ? s.samples : ka.all_wide;
    const size_t smem = std::max(ring.smem, kAloneSmem);
    auto kern = tc_list_kernel<SWB, KIND, EPI, SEED, ORDER, QSTREAM>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    CUtensorMap dmap, qmap;
    const int64_t qtiles = ((s.m + TILE - 1) / TILE + 1) / 2 * 2;
    if (SEED && ORDER == STORED) {
        ka.sample = sample_rows(s.n, rows, s.samples);
        e = sample_map(s.dt, rows, SWB, ka.kblocks, ka.sample.q, &dmap);
    } else {
        e = line_map(s.dt, ka.all_wide * 2 * rows * s.row_bytes, int64_t(ka.group) * rows * SWB, &dmap);
    }
    if (e == cudaSuccess) e = line_map(s.qt, qtiles * TILE * s.row_bytes, int64_t(ka.group) * TILE * SWB, &qmap);
    if (e != cudaSuccess) return e;
    return launch_early(kern, dim3(unsigned(qtiles), unsigned(s.splits)), kThreads, smem, st, ka, dmap, qmap);
}

template <int SWB, int KIND, int EPI, bool SEED, int ORDER = STORED>
cudaError_t launch_list_t(const ListScan &s, cudaStream_t st) {
    const Ring ring = list_ring(s.row_bytes, SWB, EPI);
    if (ring.stages == 0) return cudaErrorInvalidValue;
    if constexpr (SWB == 128 && KIND != FP4) {
        if (ring.qstream) return launch_list_q<SWB, KIND, EPI, SEED, ORDER, true>(s, ring, st);
    }
    if (ring.qstream) return cudaErrorInvalidValue;
    return launch_list_q<SWB, KIND, EPI, SEED, ORDER, false>(s, ring, st);
}

// BF16 tiles with 64-byte K-blocks, the form that allknn orders.
template <int EPI, bool SEED>
cudaError_t launch_list_order(const ListScan &s, cudaStream_t st) {
    if (!s.perm) return launch_list_t<64, BF16, EPI, SEED>(s, st);
    if (SEED || s.splits == 1) return launch_list_t<64, BF16, EPI, SEED, LOCAL>(s, st);
    return launch_list_t<64, BF16, EPI, SEED, LOCAL_SHARED>(s, st);
}

template <bool SEED>
cudaError_t launch_list_any(const ListScan &s, cudaStream_t st) {
    if (s.epi == LIST_HAMMING)
        return s.swb == 128 ? launch_list_t<128, FP4, EPI_HAM, SEED>(s, st) : cudaErrorInvalidValue;
    if (s.swb == 128) {
        if (s.epi == LIST_SCALE)
            return s.fp8 ? launch_list_t<128, FP8, EPI_SCALE, SEED>(s, st) : launch_list_t<128, BF16, EPI_SCALE, SEED>(s, st);
        if (s.epi == LIST_AFFINE && s.fp8) return launch_list_t<128, FP8, EPI_AFF, SEED>(s, st);
        if (s.epi == LIST_SQ && !s.fp8) return launch_list_t<128, BF16, EPI_SQ, SEED>(s, st);
        return cudaErrorInvalidValue;
    }
    switch (s.epi) {
        case LIST_DOT: return launch_list_order<EPI_DOT, SEED>(s, st);
        case LIST_SQ: return launch_list_order<EPI_SQ, SEED>(s, st);
        case LIST_COS: return launch_list_order<EPI_COS, SEED>(s, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// Four K-blocks of ring beside the query tile, and the database's lines within the
// tensor map's 32-bit coordinates.
bool list_fits(int row_bytes, int swb, int epi, int64_t n) {
    const Ring ring = list_ring(row_bytes, swb, epi);
    return ring.stages > 0 && (!ring.qstream || (swb == 128 && epi != LIST_HAMMING)) &&
           (n + 512) * row_bytes / kLine < (int64_t(1) << 31);
}

cudaError_t launch_list_seed(const ListScan &s, cudaStream_t st, int *launches) {
    cudaError_t e = launch_list_any<true>(s, st);
    if (e != cudaSuccess) return e;
    // about four groups per candidate keep the bound within a fifth of the
    // sample's own kk-th distance in rank
    const unsigned blocks = unsigned((s.m + 3) / 4);
    auto bound = s.per_tile == 64 && s.kk <= 256 ? seed_bound_kernel<32>
                 : s.kk <= 64                    ? seed_bound_kernel<8>
                 : s.kk <= 160                   ? seed_bound_kernel<20>
                                                 : seed_bound_kernel<60>;
    if (launches) *launches += 2;
    return launch_early(bound, dim3(blocks), 128, 0, st, s.minima, s.m, s.groups, s.kk, s.bound);
}

cudaError_t launch_list_scan(const ListScan &s, cudaStream_t st, int *launches) {
    if (launches) *launches += 1;
    return launch_list_any<false>(s, st);
}

int sketch_row_bytes(int64_t words) { return int((words + 3) / 4 * 128); }
int sketch_tile_rows(bool queries) { return queries ? TILE : db_rows(FP4); }

cudaError_t launch_sketch_tiles(const uint64_t *x, int64_t rows, int64_t words, bool queries, int64_t tiles, uint8_t *out,
                                cudaStream_t st, int *launches) {
    const int kblocks = sketch_row_bytes(words) / 128, tile_rows = sketch_tile_rows(queries);
    const int64_t total = tiles * tile_rows * kblocks * 8;
    const int64_t blocks = std::min<int64_t>((total + 255) / 256, int64_t(device_sm_count()) * 64);
    if (launches) *launches += 1;
    sketch_tile_kernel<<<unsigned(std::max<int64_t>(1, blocks)), 256, 0, st>>>(x, rows, int(words), kblocks, tile_rows,
                                                                               tiles, out);
    return cudaGetLastError();
}

}  // namespace ssg
