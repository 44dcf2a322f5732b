// rerank.cu -- exact re-scoring of candidate lists (rerank!, src/rerank.jl:22-41).
//
// For query j, the ids in row j (1-based; the first 0 ends the list, as in
// the reference) are re-evaluated with the exact distance and the valid prefix
// is sorted.  The reference sorts with sortperm and leaves the order of equal
// distances to Base.sort; here ties are ordered by id, which is one of the
// orders the reference can produce and makes the output deterministic.
#include "common.cuh"
#include "exact.cuh"
#include "finalize_shape.h"
#include "kernels.h"

#include <algorithm>
#include <climits>
#include <cmath>

namespace ssg {

// ---------------------------------------------------------------------------
// Finalize: select a query's best keys among its candidate segments, re-rank
// them with the exact FP32 distance (RERANK) and write the k best in
// (distance, id) order.
//
// What bounds it: for many queries the gather of the candidates' rows (C2:
// 1e6 queries x 50 rows x 384 bytes = 19.2 GB); for few queries the latency
// of one block.  So nothing here sorts the candidates: the `need` smallest of
// a query's unique 64-bit keys are selected by their bits (bisection in a
// warp, 8 bits at a time by histogram in a block), the rows of the selected
// candidates stream through shared memory 32 dimensions at a time (coalesced
// cp.async copies, three or four steps in flight), one thread then walks each
// candidate's sequential fma chain, and the order is found by counting the
// smaller keys.  Two shapes: a warp per query (up to 256 keys in, 64 out:
// allknn and ordinary batches, where a block per query left most threads idle
// at its barriers), a block per query beyond.  Against the block-wide bitonic sorts
// with a thread per gathered row that stood here: C1's 1,000 queries x 684
// keys 71 us (with the query norms' own launch) -> 26 us, one query of 5,472
// keys 171 -> 21 us, 4,096 queries x 125 rows of 768 dimensions 1,229 ->
// 391 us, C2's 1e6 queries x 50 rows of 96 10.2 -> 6.5 ms (3.0 TB/s of
// gathered rows).  The block shape gathers lists in one flat pass and selects
// by an 8-bit histogram; while it walked list after list and counted bit by
// bit, those two took most of it (64 queries of 152 lists: 16,000 and 37,000
// cycles): hamming, 64 queries x 1,550 keys 34 -> 20 us, 777 queries x 400
// keys, 44 rows of 300 30 -> 21 us, 20,000 x 1,060 keys, 115 rows of 768
// 2,640 -> 1,850 us.
// ---------------------------------------------------------------------------
namespace {

constexpr int kWarpOut = 64;               // candidates re-ranked per query in the warp shape
constexpr int kWarpsPerBlock = 4;
constexpr int kBlockThreads = 256;
constexpr int kBlockRows = 128;            // candidates staged together in the block shape
constexpr int kBlockStages = 4;
constexpr int kBlockStagesFew = 8;         // few queries: nothing else hides the rows' latency
constexpr int kFlatSegs = 512;             // lists per query whose keys a block gathers in one pass
constexpr int kMinSel = kFlatSegs / 4;     // sel and out together hold an int per list

// Length of a candidate row: the ids before its first 0 (by a block).
__device__ __forceinline__ int valid_prefix(const uint32_t *rid, int len) {
    __shared__ int valid;
    if (threadIdx.x == 0) valid = len;
    __syncthreads();
    for (int i = threadIdx.x; i < len; i += blockDim.x)
        if (rid[i] == 0) atomicMin(&valid, i);
    __syncthreads();
    return valid;
}

struct RowSource {
    const float *db, *q;  // database rows, this query's row
    int dim;
    bool vec;             // 16-byte copies: dim % 4 == 0 and both bases 16-byte aligned
};

// Copies dimensions [c0, c0 + kDimStep) of `rows` candidate rows (ids key_id0(sel[r]))
// and of the query (row `rows`) into buf, `threads` threads taking part.
__device__ __forceinline__ void stage_rows(const RowSource &s, const uint64_t *sel, int rows, int c0, float *buf,
                                           int tid, int threads) {
    if (s.vec) {
        constexpr int per = kDimStep / 4;
        for (int e = tid; e < (rows + 1) * per; e += threads) {
            const int r = e / per, c = c0 + 4 * (e % per);
            if (c >= s.dim) continue;
            const float *src = (r < rows ? s.db + size_t(key_id0(sel[r])) * s.dim : s.q) + c;
            const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(buf + r * kRowStride + (c - c0)));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
        }
    } else {
        for (int e = tid; e < (rows + 1) * kDimStep; e += threads) {
            const int r = e / kDimStep, c = c0 + e % kDimStep;
            if (c >= s.dim) continue;
            const float *src = (r < rows ? s.db + size_t(key_id0(sel[r])) * s.dim : s.q) + c;
            const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(buf + r * kRowStride + (c - c0)));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
        }
    }
}

// Continues the sequential chain of one staged row over `dims` dimensions:
// squared difference or product, in index order, one fma each.  qs = 0 turns
// the squared difference into the row's own square (the query's |q|^2).
template <int METRIC>
__device__ __forceinline__ float chain_step(float acc, const float *x, const float *q, int dims, float qs) {
    auto one = [&](float a, float b) {
        if constexpr (METRIC == SQL2 || METRIC == L2) {
            const float m = a - b * qs;
            acc = fmaf(m, m, acc);
        } else {
            acc = fmaf(a, b, acc);
        }
    };
    if (dims == kDimStep) {
#pragma unroll
        for (int c = 0; c < kDimStep; c += 4) {
            const float4 a = *reinterpret_cast<const float4 *>(x + c);
            const float4 b = *reinterpret_cast<const float4 *>(q + c);
            one(a.x, b.x); one(a.y, b.y); one(a.z, b.z); one(a.w, b.w);
        }
    } else {
        for (int c = 0; c < dims; ++c) one(x[c], q[c]);
    }
    return acc;
}

template <int METRIC>
__device__ __forceinline__ float chain_distance(float acc, uint32_t id0, const float *xn, float qn) {
    if constexpr (METRIC == SQL2) return acc;
    if constexpr (METRIC == L2) return sqrtf(acc);
    if constexpr (METRIC == NORMCOSINE) return 1.0f - acc;
    if constexpr (METRIC == IP) return -acc;
    return 1.0f - acc / (xn[id0] * qn);
}

// Completeness of an approximate candidate list.  An object y left out was
// either dropped by a full heap (or a merge of segments), so its approximate
// key a(y) is at least that segment's last key, or sits in a segment behind
// the re-ranked list: a(y) >= a_low = min(last key of every full segment,
// last re-ranked key).  Its exact FP32 distance D(y) >= a(y) + c - E, where
// c turns keys into distances and E bounds the approximation and evaluation
// errors:
//   check 1 (keys |x|^2 - 2 x.q of SqL2 / L2): c = |q|^2,
//           E = err_scale (R + |q|)^2, R a bound on |y| for every y
//           that could rank at or before the take-th candidate:
//           |y - q|^2 <= D_take (up to the FP32 evaluation's relative
//           error t^2 = (d + 2) 2^-24 of (|y| + |q|)^2) gives
//           |y| <= ((1 + t) |q| + sqrt(D_take)) / (1 - t), and
//           |y| <= sqrt(max |x|^2) always;
//   check 2 (keys -x.q): c = 1 for NormCosine, 0 for InnerProduct,
//           E = err_scale sqrt(max |x|^2) |q| + 2^-22;
//   check 3 (Cosine's keys -x.q / |x|): distances 1 + a / |q|, so
//           a_low enters as 1 + a_low / |q| and E = err_scale (the
//           split's c plus the FP32 dot, norms, division and
//           subtraction, (2 d + 16) 2^-24, all relative to 1).
// If a_low + c - E exceeds the exact distance of the take-th re-ranked
// candidate (for L2 its square, widened by 2^-20 so that sqrt rounding
// cannot tie), y ranks behind it: the list holds the exact top `take`.
// Evaluated in double.  A list shorter than asked for (heaps that a shared
// bound kept from filling) holds every candidate no heap dropped: a_low is
// then the full segments' smallest last key alone.  A list that holds every
// row needs no check (the caller's business); one shorter than `take`
// cannot be certified.  low: a_low's key, KEY_EMPTY if there is none.
template <int METRIC>
__device__ bool list_complete(const FinalizeArgs &f, int nv, uint64_t low, double qs, double q_abs, float d_take) {
    const int take = f.k_out + (f.exclude_self ? 1 : 0);
    if (nv < take || low == KEY_EMPTY) return false;
    const double xm = f.x_max;
    double dtake = double(d_take);
    if (METRIC == L2) dtake = dtake * dtake * (1.0 + 9.5367431640625e-7);
    double c, E;
    if (f.check == 1) {
        double r = xm + q_abs;
        if (dtake >= 0.0) r = fmin(xm, ((1.0 + f.err_t) * q_abs + sqrt(dtake)) / (1.0 - f.err_t)) + q_abs;
        c = qs;
        E = double(f.err_scale) * r * r;
    } else if (f.check == 3) {
        c = 1.0;
        E = double(f.err_scale);
    } else {
        c = METRIC == NORMCOSINE ? 1.0 : 0.0;
        E = double(f.err_scale) * xm * q_abs + 2.384185791015625e-7;
    }
    const double a_low = f.check == 3 ? double(key_dist(low)) / q_abs : double(key_dist(low));
    return a_low + c - E > dtake;
}

// Writes the result row from the sorted keys: the object itself left out when
// exclude_self finds it among the first k_out + 1, 0 / +Inf past the end.
// `at` is the calling thread's number of `threads`; self_pos (a place in
// sorted, or a large number) comes from the caller.
__device__ __forceinline__ void write_row(const FinalizeArgs &f, int64_t j, const uint64_t *sorted, int nv,
                                          int self_pos, int at, int threads) {
    uint32_t *oi = f.out_ids + size_t(j) * f.k_out;
    float *od = f.out_dists + size_t(j) * f.k_out;
    for (int w = at; w < f.k_out; w += threads) {
        const int i = w + (self_pos <= w ? 1 : 0);
        const uint64_t key = i < nv ? sorted[i] : KEY_EMPTY;
        oi[w] = key == KEY_EMPTY ? 0u : key_id0(key) + 1;
        od[w] = key == KEY_EMPTY ? INFINITY : key_dist(key);
    }
}

__device__ __forceinline__ uint32_t self_id(const FinalizeArgs &f, int64_t j) {
    return f.query_ids ? f.query_ids[j] : uint32_t(f.self_ids ? f.self_ids[j] : j + f.self_base);
}

// Where query j's row, flag and results are.
__device__ __forceinline__ int64_t query_row(const FinalizeArgs &f, int64_t j) {
    return f.query_ids ? int64_t(f.query_ids[j]) : j;
}

__device__ __forceinline__ uint64_t warp_min64(uint64_t v) {
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
        if (w < v) v = w;
    }
    return v;
}
__device__ __forceinline__ uint64_t warp_max64(uint64_t v) {
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
        if (w > v) v = w;
    }
    return v;
}

// Keeps the `need` smallest of a warp's `have` unique keys, need < have <= 32 *
// kWarpKeys, in the first places of s and returns a limit that they, and no
// others, are below.  (From registers, and as soon as they would be full: a
// pass over up to 1,026 keys in shared memory per bit took 548 us where this
// takes 380, 40,000 queries of clusters of 100.)
__device__ __noinline__ uint64_t keep_smallest(uint64_t *s, int have, int need) {
    const int lane = threadIdx.x % 32;
    uint64_t key[kWarpKeys];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kWarpKeys; ++i) key[i] = i * 32 + lane < have ? s[i * 32 + lane] : KEY_EMPTY;
    const uint64_t below = warp_limit<kWarpKeys>(key, need);
    __syncwarp();
    int base = 0;
#pragma unroll
    for (int i = 0; i < kWarpKeys; ++i) {
        const uint32_t vote = __ballot_sync(0xffffffffu, key[i] < below);
        if (key[i] < below) s[base + __popc(vote & ((1u << lane) - 1u))] = key[i];
        base += __popc(vote);
    }
    __syncwarp();
    return below;
}

// A warp per query: its segs * kk <= 32 * kWarpKeys keys in registers.
template <int METRIC, bool RERANK>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
finalize_warp_kernel(FinalizeArgs f, const float *__restrict__ db, const float *__restrict__ db_norm, int64_t dim,
                     const float *__restrict__ q, const float *__restrict__ q_norm, int need, int vec) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t s_sel[kWarpsPerBlock][kWarpOut];
    __shared__ uint64_t s_key[kWarpsPerBlock][kWarpOut];
    // the certificates of the block's queries, evaluated side by side: one
    // lane alone would hold the FP64 pipe for as long as eight
    __shared__ uint64_t s_low[kWarpsPerBlock];
    __shared__ float s_qsq[kWarpsPerBlock], s_take[kWarpsPerBlock];
    __shared__ int s_nv[kWarpsPerBlock];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int64_t j = int64_t(blockIdx.x) * kWarpsPerBlock + warp;
    const bool live = j < f.m;
    uint64_t *sel = s_sel[warp], *out = s_key[warp];
    griddep_wait();
    if (live) {
        const int64_t jr = query_row(f, j);
        int total = f.segs * f.kk;
        const uint64_t *src = f.cand + size_t(j) * total;
        uint64_t key[kWarpKeys];
        const uint64_t *held = nullptr;
        if (f.counts) {
            // lists: the keys within the bound gather in the ring's memory, as
            // many as the registers hold; when it is full the `need` smallest
            // so far stay and later keys have to be below them
            const int *cn = f.counts + size_t(j) * f.segs;
            const uint64_t *lists = f.cand + size_t(j) * f.segs * f.list_cap;
            const uint32_t bound = f.list_bound[j];
            constexpr int room = 32 * kWarpKeys;  // (warp_room holds it)
            uint64_t *scratch = reinterpret_cast<uint64_t *>(smem) + size_t(warp) * warp_room(need);
            uint64_t below = KEY_EMPTY;
            int have = 0;
            auto push = [&](uint64_t k) {
                if (uint32_t(k >> 32) > bound) k = KEY_EMPTY;
                uint32_t vote = __ballot_sync(0xffffffffu, k < below);
                if (have + __popc(vote) > room) {
                    below = keep_smallest(scratch, have, need);
                    have = need;
                    vote = __ballot_sync(0xffffffffu, k < below);
                }
                if (k < below) scratch[have + __popc(vote & ((1u << lane) - 1u))] = k;
                have += __popc(vote);
            };
            if (f.segs >= 8) {
                // the keys of 32 lists side by side (a lane along each list
                // waits for one load after another where a cluster fills a
                // few of them)
                for (int s0 = 0; s0 < f.segs; s0 += 32) {
                    const int c = s0 + lane < f.segs ? cn[s0 + lane] : 0;
                    int first = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(0xffffffffu, first, o);
                        if (lane >= o) first += v;
                    }
                    const int all = __shfl_sync(0xffffffffu, first, 31);
                    first -= c;
                    for (int i0 = 0; i0 < all; i0 += 32) {
                        const int i = i0 + lane;
                        int l = 0;
#pragma unroll
                        for (int step = 16; step > 0; step >>= 1)
                            if (__shfl_sync(0xffffffffu, first, l + step) <= i) l += step;
                        const int at = i - __shfl_sync(0xffffffffu, first, l);
                        push(i < all ? lists[size_t(s0 + l) * f.list_cap + at] : KEY_EMPTY);
                    }
                }
            } else {
                for (int s = 0; s < f.segs; ++s) {
                    const int c = cn[s];
                    const uint64_t *l = lists + size_t(s) * f.list_cap;
                    for (int i0 = 0; i0 < c; i0 += 32) push(i0 + lane < c ? l[i0 + lane] : KEY_EMPTY);
                }
            }
            __syncwarp();
            held = scratch;
            total = have;
        }
        int cnt = 0;
#pragma unroll
        for (int i = 0; i < kWarpKeys; ++i) {
            const int at = i * 32 + lane;
            key[i] = at >= total ? KEY_EMPTY : held ? held[at] : src[at];
            if (RERANK && int64_t(key_id0(key[i])) >= f.n_rows) key[i] = KEY_EMPTY;
            cnt += key[i] != KEY_EMPTY;
        }
        const int nvt = __reduce_add_sync(0xffffffffu, cnt);
        __syncwarp();
        uint64_t low = KEY_EMPTY;
        if (RERANK && f.check && !f.counts) {
            for (int s = lane; s < f.segs; s += 32) low = min(low, src[size_t(s) * f.kk + f.kk - 1]);
            low = warp_min64(low);
        }
        const int nv = min(need, nvt);
        // every selected key is below it
        const uint64_t below = nvt > need ? warp_limit<kWarpKeys>(key, need) : KEY_EMPTY;
        int base = 0;
#pragma unroll
        for (int i = 0; i < kWarpKeys; ++i) {
            const bool take = key[i] < below;
            const uint32_t vote = __ballot_sync(0xffffffffu, take);
            const int at = base + __popc(vote & ((1u << lane) - 1u));
            if (take && at < need) sel[at] = key[i];
            base += __popc(vote);
        }
        __syncwarp();
        uint64_t k0 = KEY_EMPTY, k1 = KEY_EMPTY;  // this lane's candidates lane, lane + 32
        if (lane < nv) k0 = sel[lane];
        if (lane + 32 < nv) k1 = sel[lane + 32];
        if constexpr (RERANK) {
            if (f.check && nv == need) {
                uint64_t last = lane < nv ? k0 : 0;
                if (lane + 32 < nv) last = max(last, k1);
                low = min(low, warp_max64(last));
            }
            // the query's row is staged behind the candidates; the lane of
            // that row sums |q|^2 for the certificate
            const int rows_s = need + 1;
            float *ring = reinterpret_cast<float *>(smem) + size_t(warp) * 2 * warp_room(need);
            const RowSource rs{db, q + size_t(jr) * dim, int(dim), vec != 0};
            const int steps = (int(dim) + kDimStep - 1) / kDimStep;
            float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
            const float s0 = lane == nv ? 0.0f : 1.0f, s1 = lane + 32 == nv ? 0.0f : 1.0f;
#pragma unroll
            for (int p = 0; p < kWarpStages - 1; ++p) {
                if (p < steps) stage_rows(rs, sel, nv, p * kDimStep, ring + size_t(p) * rows_s * kRowStride, lane, 32);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            for (int c = 0; c < steps; ++c) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kWarpStages - 2) : "memory");
                __syncwarp();
                const int nx = c + kWarpStages - 1;
                if (nx < steps)
                    stage_rows(rs, sel, nv, nx * kDimStep, ring + size_t(nx % kWarpStages) * rows_s * kRowStride, lane,
                               32);
                asm volatile("cp.async.commit_group;" ::: "memory");
                const float *buf = ring + size_t(c % kWarpStages) * rows_s * kRowStride;
                const float *qr = buf + nv * kRowStride;
                const int dims = min(kDimStep, int(dim) - c * kDimStep);
                if (lane <= nv) a0 = chain_step<METRIC>(a0, buf + lane * kRowStride, qr, dims, s0);
                if (lane + 32 <= nv) a1 = chain_step<METRIC>(a1, buf + (lane + 32) * kRowStride, qr, dims, s1);
                if (nv == 64 && lane == 0) a2 = chain_step<METRIC>(a2, qr, qr, dims, 0.0f);
            }
            const float qn = METRIC == COSINE ? q_norm[jr] : 0.0f;
            if (k0 != KEY_EMPTY) k0 = make_key(chain_distance<METRIC>(a0, key_id0(k0), db_norm, qn), key_id0(k0));
            if (k1 != KEY_EMPTY) k1 = make_key(chain_distance<METRIC>(a1, key_id0(k1), db_norm, qn), key_id0(k1));
            if (lane == nv) s_qsq[warp] = a0;
            if (lane + 32 == nv) s_qsq[warp] = a1;
            if (nv == 64 && lane == 0) s_qsq[warp] = a2;
            __syncwarp();
            sel[lane] = k0;
            if (lane + 32 < kWarpOut) sel[lane + 32] = k1;
            __syncwarp();
        }
        // place by counting the smaller keys (ids make them unique)
        int r0 = 0, r1 = 0;
        for (int i = 0; i < nv; ++i) {
            const uint64_t v = sel[i];
            r0 += v < k0;
            r1 += v < k1;
        }
        __syncwarp();
        if (lane < nv) out[r0] = k0;
        if (lane + 32 < nv) out[r1] = k1;
        __syncwarp();
        int self_pos = INT_MAX;
        if (f.exclude_self) {
            const uint32_t id = self_id(f, j);
            const int limit = min(nv, f.k_out + 1);
            for (int i = lane; i < limit; i += 32)
                if (key_id0(out[i]) == id) self_pos = i;
            self_pos = __reduce_min_sync(0xffffffffu, self_pos);
        }
        write_row(f, jr, out, nv, self_pos, lane, 32);
        if (RERANK && f.check && lane == 0) {
            const int take = f.k_out + (f.exclude_self ? 1 : 0);
            s_low[warp] = low;
            s_nv[warp] = nv;
            s_take[warp] = nv >= take ? key_dist(out[take - 1]) : 0.0f;
        }
    }
    if constexpr (RERANK) {
        if (!f.check) return;
        __syncthreads();
        const int64_t jq = int64_t(blockIdx.x) * kWarpsPerBlock + threadIdx.x;
        if (threadIdx.x < kWarpsPerBlock && jq < f.m) {
            const int nv = s_nv[threadIdx.x];
            if (int64_t(nv) < f.n_total &&
                !list_complete<METRIC>(f, nv, s_low[threadIdx.x], double(s_qsq[threadIdx.x]),
                                       sqrt(double(s_qsq[threadIdx.x])), s_take[threadIdx.x])) {
                f.flags[query_row(f, jq)] = 1;
                atomicAdd(f.flag_count, 1);
            }
        }
    }
}

// Exact keys out[i] of the rows key_id0(sel[i]), i < nv, by a block: up to
// kBlockRows rows at a time stream through the ring (rows_s of kRowStride
// floats per stage: the rows and, behind them, the query), one thread per row
// and chain.  *q_sq (not null): the query's own squares.  Ends with a barrier.
template <int METRIC, int STAGES>
__device__ __forceinline__ void block_distances(const RowSource &rs, const uint64_t *sel, int nv, uint64_t *out,
                                                float *ring, int rows_s, const float *db_norm, float qn, float *q_sq) {
    const int tid = threadIdx.x;
    const int steps = (rs.dim + kDimStep - 1) / kDimStep;
    for (int r0 = 0; r0 < nv || r0 == 0; r0 += kBlockRows) {
        const int rows = min(kBlockRows, nv - r0);
        float acc = 0.0f;
        const float qs = tid == rows ? 0.0f : 1.0f;
#pragma unroll
        for (int p = 0; p < STAGES - 1; ++p) {
            if (p < steps)
                stage_rows(rs, sel + r0, rows, p * kDimStep, ring + size_t(p) * rows_s * kRowStride, tid,
                           kBlockThreads);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int c = 0; c < steps; ++c) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();
            const int nx = c + STAGES - 1;
            if (nx < steps)
                stage_rows(rs, sel + r0, rows, nx * kDimStep, ring + size_t(nx % STAGES) * rows_s * kRowStride,
                           tid, kBlockThreads);
            asm volatile("cp.async.commit_group;" ::: "memory");
            const float *buf = ring + size_t(c % STAGES) * rows_s * kRowStride;
            if (tid <= rows)
                acc = chain_step<METRIC>(acc, buf + tid * kRowStride, buf + rows * kRowStride,
                                         min(kDimStep, rs.dim - c * kDimStep), qs);
        }
        if (tid < rows) {
            const uint32_t id0 = key_id0(sel[r0 + tid]);
            out[r0 + tid] = make_key(chain_distance<METRIC>(acc, id0, db_norm, qn), id0);
        }
        if (r0 == 0 && tid == rows && q_sq) *q_sq = acc;  // the query's row: |q|^2
        __syncthreads();  // the ring is refilled
    }
}

// A block per query.  cap: room for keys in shared memory (every key of the
// query's segments; of lists with more than that, only keys below a limit
// found by counting are taken); sel_cap: room for the selected ones (0: they take the keys' place,
// when nothing is left out).
template <int METRIC, bool RERANK, int STAGES>
__global__ void __launch_bounds__(kBlockThreads)
finalize_block_kernel(FinalizeArgs f, const float *__restrict__ db, const float *__restrict__ db_norm, int64_t dim,
                      const float *__restrict__ q, const float *__restrict__ q_norm, int need, int cap, int sel_cap,
                      int vec) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *keys = reinterpret_cast<uint64_t *>(smem);
    uint64_t *sel = sel_cap ? keys + cap : keys;
    uint64_t *out = sel_cap ? sel + sel_cap : keys + cap;  // as long as sel
    float *ring = reinterpret_cast<float *>(out + (sel_cap ? sel_cap : cap));
    // where each list's keys start, then the selection's histogram, in the
    // room of the selected keys (sel_cap >= kMinSel or nothing is selected)
    int *s_pre = reinterpret_cast<int *>(sel);
    __shared__ int s_cnt[3], s_n, s_picked, s_self, s_digit, s_under, s_in;
    __shared__ int s_warp[kBlockThreads / 32];
    __shared__ unsigned long long s_min, s_max, s_low, s_last;
    __shared__ float s_qsq;
    const int tid = threadIdx.x, lane = tid % 32;
    griddep_wait();
    const int64_t j = blockIdx.x, jr = query_row(f, j);
    const int total = f.segs * f.kk;
    const uint64_t *src = f.cand + size_t(j) * total;
    if (tid == 0) {
        s_n = s_picked = 0;
        s_cnt[0] = s_cnt[1] = s_cnt[2] = 0;
        s_min = s_low = KEY_EMPTY;
        s_max = s_last = 0;
        s_self = INT_MAX;
    }
    __syncthreads();
    // the query's keys, empty slots left out (or, gathered in one pass, left
    // empty in place: `slots` of them)
    int slots = -1;
    uint64_t mn = KEY_EMPTY, mx = 0;
    auto push = [&](uint64_t key) {  // by whole warps
        if (RERANK && int64_t(key_id0(key)) >= f.n_rows) key = KEY_EMPTY;
        const bool have = key != KEY_EMPTY;
        const uint32_t vote = __ballot_sync(0xffffffffu, have);
        int base = 0;
        if (lane == 0 && vote) base = atomicAdd(&s_n, __popc(vote));
        base = __shfl_sync(0xffffffffu, base, 0);
        const int at = base + __popc(vote & ((1u << lane) - 1u));
        if (have && at < cap) {
            keys[at] = key;
            mn = min(mn, key);
            mx = max(mx, key);
        }
    };
    if (f.counts) {
        // eight lanes per list
        const int *cn = f.counts + size_t(j) * f.segs;
        const uint64_t *lists = f.cand + size_t(j) * f.segs * f.list_cap;
        const int sub = lane % 8;
        const uint32_t bound = f.list_bound[j];
        auto each_key = [&](auto &&body) {
            for (int s0 = (tid / 32) * 4; s0 < f.segs; s0 += kBlockThreads / 8) {
                const int sg = s0 + lane / 8;
                const int c = sg < f.segs ? cn[sg] : 0;
                const uint64_t *l = lists + size_t(sg) * f.list_cap;
                const int most = __reduce_max_sync(0xffffffffu, c);
                for (int i = sub; i < most + sub; i += 8) {
                    const uint64_t k = i < c ? l[i] : KEY_EMPTY;
                    body(uint32_t(k >> 32) <= bound ? k : KEY_EMPTY);
                }
            }
        };
        // two lists per thread: where each one's keys start among all
        int all;
        const bool flat = f.segs <= kFlatSegs && sel_cap;
        if (flat) {
            const int s2 = 2 * tid;
            const int c0 = s2 < f.segs ? cn[s2] : 0, c1 = s2 + 1 < f.segs ? cn[s2 + 1] : 0;
            int incl = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) s_warp[tid / 32] = incl;
            __syncthreads();
            int before = 0;
            all = 0;
#pragma unroll
            for (int w = 0; w < kBlockThreads / 32; ++w) {
                before += w < tid / 32 ? s_warp[w] : 0;
                all += s_warp[w];
            }
            s_pre[s2] = before + incl - c0 - c1;
            s_pre[s2 + 1] = before + incl - c1;
            __syncthreads();
        } else {
            int sum = 0;
            for (int s = tid; s < f.segs; s += kBlockThreads) sum += cn[s];
            sum = __reduce_add_sync(0xffffffffu, sum);
            if (lane == 0 && sum) atomicAdd(&s_cnt[0], sum);
            __syncthreads();
            all = s_cnt[0];
            __syncthreads();
            if (tid == 0) s_cnt[0] = 0;
        }
        uint64_t lim = KEY_EMPTY;
        if (all > cap) {
            // more keys than fit: a limit with at least `need` and at most
            // cap keys below it (keys are unique, so one exists).  First the
            // bound itself: where it is the distance of many (equal rows),
            // only the ids' bits are left to find (49 queries x 49,965 equal
            // FP8 rows, k = 50: 537 -> 327 us)
            __syncthreads();
            uint64_t p = 0;
            int it = 0;
            for (int b = 64; b >= 0; --b, ++it) {
                const uint64_t t = b == 64 ? uint64_t(bound) << 32 : p | (1ull << b);
                int c = 0;
                each_key([&](uint64_t key) { c += key < t; });
                c = __reduce_add_sync(0xffffffffu, c);
                if (lane == 0 && c) atomicAdd(&s_cnt[it % 3], c);
                __syncthreads();
                c = s_cnt[it % 3];
                if (tid == 0) s_cnt[(it + 2) % 3] = 0;
                if (c >= need && c <= cap) { lim = t; break; }
                if (c < need) {
                    p = t;
                    if (b == 64) b = 64 - __clzll(f.n_total);  // (ids are below 2^b)
                }
            }
            __syncthreads();
            if (tid < 3) s_cnt[tid] = 0;
            __syncthreads();
        }
        if (flat && all <= cap) {
            // one pass over all keys side by side (a group of lanes walking
            // lists in turn waits for a count, then for keys, list after list)
            slots = all;
            int have = 0;
#pragma unroll 4
            for (int i = tid; i < all; i += kBlockThreads) {
                int sg = 0;
#pragma unroll
                for (int step = kFlatSegs / 2; step > 0; step >>= 1)
                    if (sg + step < f.segs && s_pre[sg + step] <= i) sg += step;
                uint64_t key = lists[size_t(sg) * f.list_cap + (i - s_pre[sg])];
                if (uint32_t(key >> 32) > bound || (RERANK && int64_t(key_id0(key)) >= f.n_rows)) key = KEY_EMPTY;
                keys[i] = key;
                if (key != KEY_EMPTY) {
                    ++have;
                    mn = min(mn, key);
                    mx = max(mx, key);
                }
            }
            have = __reduce_add_sync(0xffffffffu, have);
            if (lane == 0 && have) atomicAdd(&s_n, have);
        } else {
            each_key([&](uint64_t key) { push(key < lim ? key : KEY_EMPTY); });
        }
    } else {
        for (int i0 = 0; i0 < total; i0 += kBlockThreads) push(i0 + tid < total ? src[i0 + tid] : KEY_EMPTY);
    }
    mn = warp_min64(mn);
    mx = warp_max64(mx);
    uint64_t low = KEY_EMPTY;
    if (RERANK && f.check && !f.counts) {
        for (int s = tid; s < f.segs; s += kBlockThreads) low = min(low, src[size_t(s) * f.kk + f.kk - 1]);
        low = warp_min64(low);
    }
    if (lane == 0) {
        atomicMin(&s_min, mn);
        atomicMax(&s_max, mx);
        if (RERANK && f.check) atomicMin(&s_low, low);
    }
    __syncthreads();
    const int nvt = min(s_n, cap);
    const int nv = min(need, nvt);
    const bool holes = slots >= 0;  // (then sel is apart from keys)
    if (!holes) slots = nvt;
    if (nvt > need || holes) {
        // the keys below `below` are the `need` smallest: the digit (8 bits
        // from the first one that differs) that the need-th falls into, by a
        // histogram, until a digit's end meets the count (a compare and count
        // per bit took 900 to 1,150 cycles for each of 6 to 40 bits)
        uint64_t below = KEY_EMPTY;
        if (nvt > need) {
            const uint64_t lo = s_min, hi = s_max;
            int bits = 64 - __clzll(lo ^ hi), rem = need;
            uint64_t p = bits >= 64 ? 0ull : lo >> bits;
            for (;;) {
                const int w = min(8, bits), shift = bits - w;
                s_pre[tid] = 0;
                __syncthreads();
                for (int i = tid; i < slots; i += kBlockThreads) {
                    const uint64_t key = keys[i];
                    if (key != KEY_EMPTY && (bits >= 64 || key >> bits == p))
                        atomicAdd(&s_pre[int(key >> shift) & ((1 << w) - 1)], 1);
                }
                __syncthreads();
                if (tid < 32) {
                    int c[8], sum = 0;
#pragma unroll
                    for (int e = 0; e < 8; ++e) sum += c[e] = s_pre[8 * tid + e];
                    int incl = sum;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += v;
                    }
                    int under = incl - sum;
                    if (under < rem && rem <= incl) {
                        bool found = false;
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            if (!found && rem <= under + c[e]) {
                                found = true;
                                s_digit = 8 * tid + e;
                                s_under = under;
                                s_in = c[e];
                            }
                            under += c[e];
                        }
                    }
                }
                __syncthreads();
                p = (p << w) | uint64_t(s_digit);
                rem -= s_under;
                bits = shift;
                if (s_in == rem || bits == 0) {
                    below = (p + 1) << bits;
                    if (below == 0) below = KEY_EMPTY;
                    break;
                }
            }
        }
        // (a count of its own: slower warps may still be reading s_n)
        for (int i0 = 0; i0 < slots; i0 += kBlockThreads) {
            const int i = i0 + tid;
            const uint64_t key = i < slots ? keys[i] : KEY_EMPTY;
            const bool take = key < below;
            const uint32_t vote = __ballot_sync(0xffffffffu, take);
            int base = 0;
            if (lane == 0 && vote) base = atomicAdd(&s_picked, __popc(vote));
            base = __shfl_sync(0xffffffffu, base, 0);
            const int at = base + __popc(vote & ((1u << lane) - 1u));
            if (take && at < need) sel[at] = key;
        }
        __syncthreads();
    } else if (sel != keys) {
        for (int i = tid; i < nv; i += kBlockThreads) sel[i] = keys[i];
        __syncthreads();
    }
    if constexpr (RERANK) {
        if (f.check && nv == need) {
            uint64_t last = 0;
            for (int i = tid; i < nv; i += kBlockThreads) last = max(last, sel[i]);
            last = warp_max64(last);
            if (lane == 0) atomicMax(&s_last, last);
            __syncthreads();
            if (tid == 0 && s_last < s_low) s_low = s_last;
        }
        const RowSource rs{db, q + size_t(jr) * dim, int(dim), vec != 0};
        block_distances<METRIC, STAGES>(rs, sel, nv, out, ring, min(need, kBlockRows) + 1, db_norm,
                                METRIC == COSINE ? q_norm[jr] : 0.0f, &s_qsq);
        uint64_t *t = sel;
        sel = out;
        out = t;
    }
    double q_abs = 0.0;
    if (RERANK && f.check && tid == 0) q_abs = sqrt(double(s_qsq));  // beside the placing
    // place by counting the smaller keys; long lists by a bitonic sort
    if (nv <= 512) {
        for (int i = tid; i < nv; i += kBlockThreads) {
            const uint64_t v = sel[i];
            int r = 0;
            for (int k = 0; k < nv; ++k) r += sel[k] < v;
            out[r] = v;
        }
        __syncthreads();
    } else {
        int P = 1024;
        while (P < nv) P <<= 1;
        for (int i = tid; i < P; i += kBlockThreads) out[i] = i < nv ? sel[i] : KEY_EMPTY;
        block_bitonic_sort(out, P);
    }
    if (f.exclude_self) {
        const uint32_t id = self_id(f, j);
        const int limit = min(nv, f.k_out + 1);
        for (int i = tid; i < limit; i += kBlockThreads)
            if (key_id0(out[i]) == id) atomicMin(&s_self, i);
        __syncthreads();
    }
    write_row(f, jr, out, nv, s_self, tid, kBlockThreads);
    if (RERANK && f.check && tid == 0 && int64_t(nv) < f.n_total) {
        const int take = f.k_out + (f.exclude_self ? 1 : 0);
        if (!list_complete<METRIC>(f, nv, s_low, double(s_qsq), q_abs, nv >= take ? key_dist(out[take - 1]) : 0.0f)) {
            f.flags[jr] = 1;
            atomicAdd(f.flag_count, 1);
        }
    }
}

template <int METRIC, bool RERANK>
cudaError_t launch_finalize_t(const FinalizeArgs &f, const float *db, const float *db_norm, int64_t dim,
                              const float *q, const float *q_norm, int need, cudaStream_t st) {
    // lists: room for twice the keys a seeded bound leaves on average
    const int total = f.counts ? std::max(f.list_keys, 2 * need) : f.segs * f.kk;
    const bool vec = RERANK && dim % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(db) | reinterpret_cast<uintptr_t>(q)) & 15) == 0;
    // (lists: a block is done sooner with few queries, and with more rows to
    // gather than lanes: 777 queries x 45 rows of 300 dimensions 30 us against
    // 38 in warps, 1,000 x 18 of 128 27.5 against 23.6; in a locality order the
    // warps share rows, 38,912 x 23 of 100 744 against 600)
    if ((f.counts ? f.m >= 256 && (f.query_ids || (need <= 32 && f.list_keys <= 1024)) : total <= 32 * kWarpKeys) &&
        need <= kWarpOut) {
        const size_t smem =
            RERANK || f.counts ? size_t(kWarpsPerBlock) * warp_room(need) * 8 : 0;
        auto kern = finalize_warp_kernel<METRIC, RERANK>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
        const unsigned blocks = unsigned((f.m + kWarpsPerBlock - 1) / kWarpsPerBlock);
        return launch_early(kern, dim3(blocks), 32 * kWarpsPerBlock, smem, st, f, db, db_norm, dim, q, q_norm, need,
                            vec ? 1 : 0);
    }
    // the sorted order of more than 512 selected keys takes a power of two
    const bool in_place = total <= need;
    int out_cap = need <= 512 ? (need + 1) / 2 * 2 : next_pow2(need);  // even: the ring behind is 16-byte aligned
    if (!in_place) out_cap = std::max(out_cap, kMinSel);
    const int cap = in_place ? std::max((total + 1) / 2 * 2, out_cap) : (total + 1) / 2 * 2;
    const size_t keys = in_place ? 2 * size_t(cap) : size_t(cap) + 2 * size_t(out_cap);
    const size_t stage = RERANK ? size_t(std::min(need, kBlockRows) + 1) * kRowStride * 4 : 0;
    size_t smem = keys * 8 + kBlockStages * stage;
    if (smem > 226 * 1024) return cudaErrorInvalidValue;
    auto kern = finalize_block_kernel<METRIC, RERANK, kBlockStages>;
    // at most a block per SM: more steps of the rows in flight (at more, the
    // other blocks of an SM hide the rows' latency and room is what counts)
    if (RERANK && f.m <= device_sm_count() && keys * 8 + kBlockStagesFew * stage <= 226 * 1024) {
        smem = keys * 8 + kBlockStagesFew * stage;
        kern = finalize_block_kernel<METRIC, RERANK, kBlockStagesFew>;
    }
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    return launch_early(kern, dim3(unsigned(f.m)), kBlockThreads, smem, st, f, db, db_norm, dim, q, q_norm, need, cap,
                        in_place ? 0 : out_cap, vec ? 1 : 0);
}

}  // namespace

cudaError_t launch_finalize(const FinalizeArgs &f, cudaStream_t st, int *launches) {
    const int need = std::min(f.counts ? f.kk : f.segs * f.kk, f.k_out + (f.exclude_self ? 1 : 0));
    if (launches) *launches += 1;
    return launch_finalize_t<SQL2, false>(f, nullptr, nullptr, 0, nullptr, nullptr, need, st);
}

cudaError_t launch_finalize_rerank(int metric, const FinalizeArgs &args, const float *db, const float *db_norm,
                                   int64_t dim, const float *q, const float *q_norm, cudaStream_t st,
                                   int *launches) {
    FinalizeArgs f = args;
    const int rr = f.rerank ? f.rerank : f.kk;
    if (rr > (f.counts ? f.kk : f.segs * f.kk)) return cudaErrorInvalidValue;
    if (launches) *launches += 1;
    f.x_max = std::sqrt(double(f.max_x_sq));
    f.err_t = std::sqrt(double(dim + 2) * 5.9604644775390625e-8);
    switch (metric) {
        case SQL2: return launch_finalize_t<SQL2, true>(f, db, db_norm, dim, q, q_norm, rr, st);
        case L2: return launch_finalize_t<L2, true>(f, db, db_norm, dim, q, q_norm, rr, st);
        case NORMCOSINE: return launch_finalize_t<NORMCOSINE, true>(f, db, db_norm, dim, q, q_norm, rr, st);
        case COSINE: return launch_finalize_t<COSINE, true>(f, db, db_norm, dim, q, q_norm, rr, st);
        case IP: return launch_finalize_t<IP, true>(f, db, db_norm, dim, q, q_norm, rr, st);
        default: return cudaErrorInvalidValue;
    }
}

namespace {

// Sketches are two words or so long: a thread per candidate.
__global__ void rerank_sketches_kernel(const void *db, int64_t dim, const void *q, int len, int P, uint32_t *ids,
                                       float *dists) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s = reinterpret_cast<uint64_t *>(smem);
    const int64_t j = blockIdx.x;
    uint32_t *rid = ids + j * len;
    float *rd = dists + j * len;
    const int nv = valid_prefix(rid, len);
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        s[i] = KEY_EMPTY;
        if (i < nv) s[i] = make_key(exact_pair<HAMMING>(db, int64_t(rid[i]) - 1, dim, q, j, nullptr, nullptr), rid[i] - 1);
    }
    block_bitonic_sort(s, P);
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
        rid[i] = key_id0(s[i]) + 1;
        rd[i] = key_dist(s[i]);
    }
}

// Rows of floats: staged through shared memory as the finalize's are, not
// read by the thread that walks the chain (32 lanes on 32 rows used one
// sector in 32 loads).  What bounds it: the gather of m * len rows (1,000 x
// 512 rows of 768: 1,298 -> 317 us, 5 TB/s).
template <int METRIC>
__global__ void __launch_bounds__(kBlockThreads)
rerank_rows_kernel(const float *__restrict__ db, const float *__restrict__ db_norm, int64_t dim,
                   const float *__restrict__ q, const float *__restrict__ q_norm, int len, int P, uint32_t *ids,
                   float *dists, int vec) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *s = reinterpret_cast<uint64_t *>(smem);
    float *ring = reinterpret_cast<float *>(s + P);
    const int64_t j = blockIdx.x;
    uint32_t *rid = ids + j * len;
    float *rd = dists + j * len;
    const int nv = valid_prefix(rid, len);
    if (nv == 0) return;
    for (int i = threadIdx.x; i < P; i += blockDim.x) s[i] = i < nv ? uint64_t(rid[i] - 1) : KEY_EMPTY;
    __syncthreads();
    const RowSource rs{db, q + size_t(j) * dim, int(dim), vec != 0};
    block_distances<METRIC, kBlockStages>(rs, s, nv, s, ring, min(len, kBlockRows) + 1, db_norm, METRIC == COSINE ? q_norm[j] : 0.0f,
                            nullptr);
    block_bitonic_sort(s, P);
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
        rid[i] = key_id0(s[i]) + 1;
        rd[i] = key_dist(s[i]);
    }
}

template <int METRIC>
cudaError_t launch_rerank_rows(const float *db, const float *db_norm, int64_t dim, const float *q, const float *q_norm,
                               int64_t m, int len, int P, uint32_t *ids, float *dists, cudaStream_t st) {
    const bool vec = dim % 4 == 0 && ((reinterpret_cast<uintptr_t>(db) | reinterpret_cast<uintptr_t>(q)) & 15) == 0;
    const size_t smem = size_t(P) * 8 + size_t(kBlockStages) * (std::min(len, kBlockRows) + 1) * kRowStride * 4;
    auto kern = rerank_rows_kernel<METRIC>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    kern<<<unsigned(m), kBlockThreads, smem, st>>>(db, db_norm, dim, q, q_norm, len, P, ids, dists, vec);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_rerank(int metric, const void *db, const float *db_norm, int64_t dim,
                          const void *q, const float *q_norm, int64_t m, int len,
                          uint32_t *ids, float *dists, cudaStream_t st, int *launches) {
    if (m <= 0 || len <= 0) return cudaSuccess;
    const int P = std::max(2, next_pow2(len));  // even: the ring behind the keys is 16-byte aligned
    if (size_t(P) * 8 > 200 * 1024) return cudaErrorInvalidValue;  // (+ 74 KB of the ring: P is at most 16,384)
    if (launches) *launches += 1;
    if (metric == HAMMING) {
        const int smem = P * 8;
        cudaError_t e = cudaFuncSetAttribute(rerank_sketches_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        rerank_sketches_kernel<<<unsigned(m), 128, smem, st>>>(db, dim, q, len, P, ids, dists);
        return cudaGetLastError();
    }
    const float *x = static_cast<const float *>(db), *y = static_cast<const float *>(q);
    switch (metric) {
        case SQL2: return launch_rerank_rows<SQL2>(x, db_norm, dim, y, q_norm, m, len, P, ids, dists, st);
        case L2: return launch_rerank_rows<L2>(x, db_norm, dim, y, q_norm, m, len, P, ids, dists, st);
        case NORMCOSINE: return launch_rerank_rows<NORMCOSINE>(x, db_norm, dim, y, q_norm, m, len, P, ids, dists, st);
        case COSINE: return launch_rerank_rows<COSINE>(x, db_norm, dim, y, q_norm, m, len, P, ids, dists, st);
        case IP: return launch_rerank_rows<IP>(x, db_norm, dim, y, q_norm, m, len, P, ids, dists, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ssg
