// Exact FP32 brute-force k-NN on CUDA cores, bit-identical to
// BruteForceIndex::search_filtered (src/brute.rs:131-160) with the AVX2
// kernels (src/kernels/x86.rs:32-131).
//
// Layout of the arithmetic: lane (c, l) = (lane >> 3, lane & 7) of a warp is
// AVX2 accumulator chain c, vector lane l, i.e. column `lane` of every 32. A
// warp scores QW queries x RW rows (64 pairs): every lane runs the FMA chain
// of its accumulator for each pair, two rows per packed f32x2 instruction;
// then a transpose-reduce adds the 32 accumulators of each pair in the
// reference order (lane bits 3, 4 = chains (c0+c1), (c2+c3), then their sum;
// bit 2 = v_l + v_{l+4}; bit 0 then bit 1 = the horizontal sum), leaving two
// rows' sums of one query in each lane.
// Each block keeps a per-query top-k (by total_cmp distance, then key) of its
// row slice; a merge kernel combines the slices.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "device.hpp"
#include "warp_sort.cuh"

namespace hnswgpu {
namespace dev {

// Top-k entries are (fkey(distance) << 32) | rank of the row's key, so the
// u64 order is the reference's (total_cmp distance, key) order. The rank is
// the row itself when the keys ascend (krank null).
__device__ __forceinline__ uint64_t brute_entry(const BruteArgs& a, float dist, uint32_t row) {
    return (uint64_t(fkey(dist)) << 32) | (a.krank ? __ldg(a.krank + row) : row);
}

// One query's top-k of a warp: an ascending list of n <= kk entries and a
// buffer of cnt <= 32 entries still to be merged into it. Entries are
// buffered so that one merge serves up to 32 of them.
struct TopList {
    uint64_t* L;
    uint64_t* B;
    uint32_t n, cnt;
};

__device__ __forceinline__ void top_flush(TopList& t, uint32_t kk) {
    const int lane = lane_id();
    const uint64_t x = uint32_t(lane) < t.cnt ? t.B[lane] : ~0ull;
    const uint64_t worst = t.n == kk ? t.L[kk - 1] : ~0ull;
    const uint32_t S = __ballot_sync(kFull, x < worst);
    t.cnt = 0;
    if (S == 0) return;
    // The buffer is free once every lane holds its entry: it is the merge's scratch.
    __syncwarp();
    batch_merge_gather(t.L, 0, t.n, S, x, kk, t.B);
    __syncwarp();
    t.n = min(t.n + uint32_t(__popc(S)), kk);
}

// Adds the entries x of the lanes in W (all lanes call); true if the buffer
// was merged into the list for it.
__device__ __forceinline__ bool top_push(TopList& t, uint32_t W, uint64_t x, uint32_t kk) {
    const uint32_t c = __popc(W);
    const bool full = t.cnt + c > 32;
    if (full) top_flush(t, kk);
    const int lane = lane_id();
    if ((W >> lane) & 1u) t.B[t.cnt + __popc(W & ((1u << lane) - 1u))] = x;
    t.cnt += c;
    __syncwarp();
    return full;
}

// vector::check + normalisation of each query (one warp per query). The f64
// squared norm adds its terms in row order, as the reference does: the
// products are formed 32 at a time, one per lane, and every lane adds them in
// order (the chain of additions is all that is serial; one lane doing both
// took 31 us for 768 dimensions). out_count and the lane minima start as "no
// bound" for the score kernel.
__global__ void brute_prep_kernel(BruteArgs a) {
    const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= a.nq) return;
    const float* src = a.queries + size_t(q) * a.dim;
    float* dst = a.qprep + size_t(q) * a.dp;
    bool bad = false;
    double norm = 0.0;
    for (uint32_t b = 0; b < a.dp; b += 32) {
        const uint32_t i = b + uint32_t(lane);
        const float x = i < a.dim ? src[i] : 0.0f;
        bad |= !isfinite(x);
        dst[i] = x;
        const double p = __dmul_rn(double(x), double(x));
        const uint32_t m = min(32u, a.dim - b);
        if (m == 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j) norm = __dadd_rn(norm, __shfl_sync(kFull, p, j));
        } else {
            for (uint32_t j = 0; j < m; ++j) norm = __dadd_rn(norm, __shfl_sync(kFull, p, int(j)));
        }
    }
    bad = __any_sync(kFull, bad);
    int32_t st = 0;
    if (bad || norm > double(3.40282346638528859812e+38F) / 8.0) st = 3;
    if (st == 0 && a.metric == 2) {
        if (norm == 0.0) st = 4;
        else {
            const double inv = __ddiv_rn(1.0, __dsqrt_rn(norm));
            for (uint32_t i = lane; i < a.dim; i += 32) dst[i] = __double2float_rn(__dmul_rn(double(dst[i]), inv));
        }
    }
    if (lane == 0) {
        a.out_status[q] = st;
        a.out_count[q] = 0xFFFFFFFFu;
    }
    if (a.minima)
        for (uint32_t i = lane; i < kBruteMinima; i += 32) a.minima[size_t(q) * kBruteMinima + i] = 0xFFFFFFFFu;
}

// Whether query q admits row r under the optional filter.
__device__ __forceinline__ bool brute_admits(const BruteArgs& a, uint32_t q, uint32_t r) {
    if (!a.filter_bits || (a.filter_used && !a.filter_used[q])) return true;
    const size_t sel = a.filter_ids ? size_t(a.filter_ids[q]) : size_t(q);
    const uint64_t* bits = a.filter_bits + (a.filter_stride ? sel * a.filter_stride : 0);
    const uint64_t bit = a.filter_by_row ? uint64_t(r) : __ldg(a.keys + r);
    return bit < a.filter_nbits && ((__ldg(bits + (bit >> 6)) >> (bit & 63)) & 1ull);
}

// The rows that one filter for the whole batch admits, in any order: the score
// kernel then reads and scores only those. (100 queries x 50k x 100 rows with
// 20 % admitted: testing the bit after scoring every row took 229 us a call.)
__global__ void __launch_bounds__(256) brute_rows_kernel(BruteArgs a) {
    __shared__ uint32_t base, wcount[8];
    const uint32_t r = blockIdx.x * 256 + threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool in = r < a.n && brute_admits(a, 0, r);
    const uint32_t M = __ballot_sync(kFull, in);
    if (lane == 0) wcount[warp] = __popc(M);
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t w = 0; w < 8; ++w) {
        before += w < warp ? wcount[w] : 0u;
        all += wcount[w];
    }
    if (threadIdx.x == 0 && all) base = atomicAdd(a.row_list, all);
    __syncthreads();
    if (in) a.row_list[1 + base + before + __popc(M & ((1u << lane) - 1u))] = r;
}

// Two f32 operations per instruction, each rounded as its scalar form.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// acc += (q + r)^2 (L2: q is staged negated, and (r - q)^2 is (q - r)^2 bit
// for bit) or q * r, element by element.
template <bool L2>
__device__ __forceinline__ void acc_pair(uint64_t& acc, uint64_t q, uint64_t r) {
    if (L2) {
        const uint64_t d = add2(q, r);
        asm("fma.rn.f32x2 %0, %1, %1, %0;" : "+l"(acc) : "l"(d));
    } else {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(q), "l"(r));
    }
}

// One stage of the transpose-reduce: of the first N accumulators a lane keeps
// half and adds the partner lane's values of the same pairs. With PERM the
// lane's accumulators are laid out so that it always keeps the lower half
// (the queries were read in an order that depends on the lane); otherwise its
// lane bit selects the half.
template <int N, bool PERM, int ALL>
__device__ __forceinline__ void fold_pairs(uint64_t (&v)[ALL], int bit, bool hi) {
#pragma unroll
    for (int p = 0; p < N / 2; ++p) {
        const uint64_t send = !PERM && hi ? v[p] : v[p + N / 2];
        const uint64_t keep = !PERM && hi ? v[p + N / 2] : v[p];
        v[p] = add2(keep, __shfl_xor_sync(kFull, send, bit));
    }
}

// Shape of the score kernel: WQ x WR warps, each scoring QW queries x RW rows
// (64 pairs) of the block's tile of QB queries x RB rows. Rows stream through
// a ring of kStages chunks of KC columns filled by cp.async; the queries stay
// in shared memory, chunk by chunk. Row strides are padded by four floats so
// that a column of rows spreads over the banks (the scalar tail reads one;
// the queries' tails have a padded array of their own).
template <int QW_, int RW_, int WQ_, int WR_>
struct BruteTile {
    static constexpr int QW = QW_, RW = RW_, WQ = WQ_, WR = WR_;
    static constexpr int QB = QW * WQ, RB = RW * WR, kWarps = WQ * WR, kThreads = 32 * kWarps;
    // With one warp along the queries a row belongs to one warp, which then
    // copies its own rows and waits for nobody else.
    static constexpr bool kPrivate = WQ == 1;
    static constexpr int KC = RB >= 128 ? 32 : (RB >= 32 ? 64 : 128);
    static constexpr int kStages = kPrivate ? 4 : 3;
    static constexpr int kRowStride = KC + 4;
    static constexpr size_t kRingBytes = size_t(kStages) * RB * kRowStride * 4;
    static constexpr size_t kBufBytes = size_t(kWarps) * QW * 32 * 8;
    static constexpr int kTailStride = 9;  // tail columns (at most 7) of a query
    static size_t smem(uint32_t dp, uint32_t list_kk) {
        return size_t((dp + KC - 1) / KC) * QB * KC * 4 + size_t(QB) * kTailStride * 4 + kRingBytes + kBufBytes +
               size_t(kWarps) * QW * (size_t(list_kk) * 8 + 8);
    }
};

// Lists longer than this live in the partial-result array instead of shared
// memory (a list is only touched by a merge of up to 32 entries).
constexpr uint32_t kSharedListMax = 128;

// Smallest x (to 1/4096 of the range below hi) such that at least k of the
// values v (M per lane, of four neighboring lanes together) are <= x; hi when
// there are fewer.
template <int M>
__device__ __forceinline__ uint32_t kth_bound(const uint32_t (&v)[M], uint32_t k, uint32_t hi) {
    hi = min(hi, __shfl_xor_sync(kFull, hi, 1));
    hi = min(hi, __shfl_xor_sync(kFull, hi, 2));
    uint32_t lo = hi;
#pragma unroll
    for (int i = 0; i < M; ++i) lo = min(lo, v[i]);
    lo = min(lo, __shfl_xor_sync(kFull, lo, 1));
    lo = min(lo, __shfl_xor_sync(kFull, lo, 2));
    // `hi` is a bound (or the one given), below `lo` there are fewer than k.
#pragma unroll 1
    for (int it = 0; it < 12; ++it) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < M; ++i) c += v[i] <= mid ? 1u : 0u;
        c += __shfl_xor_sync(kFull, c, 1);
        c += __shfl_xor_sync(kFull, c, 2);
        if (c >= k) hi = mid;
        else lo = mid;
    }
    return hi;
}

// Scores every row of a slice against the block's queries and keeps each
// query's best kk. An entry costs about as much to insert as a tile of pairs
// to score, so the lists share bounds per query; a distance above one cannot
// be among the best kk. One bound is the smallest kk-th distance of any list
// (out_count, atomicMin). The other, which works long before the lists are
// full, comes from the minima of the lanes: the lanes that finish a query's
// pairs see disjoint rows, so the kk-th smallest of their minima bounds the
// kk-th distance of all. They are published and read after 1, 3, 7, ... tiles
// (a reader may see some of them late: every value is a real row's distance).
//
// What bounds it: instruction issue. A tile of 64 pairs at D = 128 takes 656
// instructions, of them 284 packed FMAs and additions (the FMA pipe is 52 %
// busy), 67 shared loads and 63 shuffles. 1,000 queries x 100k x 128 (L2, k =
// 10): 1.66 ms; with scalar FMAs on 4 x 8 pairs, copies that did not overlap
// and single insertions 3.47 ms; eight lanes per pair (16-byte shared loads)
// 1.95 ms, bound by the shared-memory pipe, which serves a quarter warp at a
// time; 16 rows per warp 2.34 ms, eight warps per SM not hiding latency; three
// blocks per SM instead of four 1.72 ms.
// LIST: the rows of a.row_list instead of all.
template <bool L2, class T, bool LIST>
__global__ void __launch_bounds__(T::kThreads, T::kThreads == 128 ? 4 : 8) brute_score_kernel(BruteArgs a, uint32_t kk,
                                                                                            uint32_t rows_per,
                                                                                            uint32_t nslices) {
    constexpr int QW = T::QW, RW = T::RW, RP = RW / 2, NP = QW * RP;
    static_assert(NP == 32, "a lane ends with one packed pair of rows of one query");
    static_assert((T::QB * T::kTailStride) % 2 == 0, "8-byte alignment of the lists");
    extern __shared__ __align__(16) char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wq = warp % T::WQ, wr = warp / T::WQ;
    const uint32_t dp = a.dp;
    const uint32_t nk = (dp + T::KC - 1) / T::KC;
    const bool shared_lists = kk <= kSharedListMax;
    float* sq = reinterpret_cast<float*>(smem);
    float* sr = sq + size_t(nk) * T::QB * T::KC;
    float* sqt = sr + T::kRingBytes / 4;
    uint64_t* bufs = reinterpret_cast<uint64_t*>(sqt + T::QB * T::kTailStride);
    uint2* meta = reinterpret_cast<uint2*>(reinterpret_cast<char*>(bufs) + T::kBufBytes);  // per list: (n, cnt)
    uint64_t* lists = reinterpret_cast<uint64_t*>(meta + T::kWarps * QW);
    const uint32_t q0 = blockIdx.x * T::QB, slice = blockIdx.y;
    // Positions of the row list (its count first) when there is one, else rows.
    const uint32_t* list = LIST ? a.row_list + 1 : nullptr;
    const uint32_t nrows = LIST ? *a.row_list : a.n;
    if (LIST) rows_per = ((nrows + nslices - 1) / nslices + T::RB - 1) / T::RB * T::RB;
    const uint32_t r_begin = min(nrows, slice * rows_per), r_end = min(nrows, r_begin + rows_per);
    const uint32_t wq0 = q0 + uint32_t(wq * QW);  // this warp's first query
    const bool active = wq0 < a.nq;
    uint64_t* wbuf = bufs + size_t(warp) * QW * 32;
    uint2* wmeta = meta + warp * QW;
    // The list of warp w's query i: shared memory, or (one warp per query
    // then, T::WR == 1) the slice's list in the partial-result array.
    auto list_of = [&](int w, int i) -> uint64_t* {
        if (shared_lists) return lists + (size_t(w) * QW + i) * kk;
        const uint32_t q = min(q0 + uint32_t((w % T::WQ) * QW + i), a.nq - 1);
        return a.part + (size_t(q) * nslices + slice) * kk;
    };
    for (uint32_t i = threadIdx.x; i < T::QB * (dp >> 2); i += T::kThreads) {
        const uint32_t qq = i / (dp >> 2), j = (i % (dp >> 2)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q0 + qq < a.nq) v = *reinterpret_cast<const float4*>(a.qprep + size_t(q0 + qq) * dp + j);
        if (L2) v = make_float4(-v.x, -v.y, -v.z, -v.w);
        *reinterpret_cast<float4*>(sq + (j / T::KC * T::QB + qq) * T::KC + j % T::KC) = v;
    }
    if (lane < QW) wmeta[lane] = make_uint2(0, 0);
    const uint32_t nfull = a.dim >> 5, rem8 = (a.dim & 31) >> 3, tail0 = (nfull << 5) + (rem8 << 3);
    const uint32_t ntail = a.dim - tail0;
    for (uint32_t i = threadIdx.x; i < T::QB * 8; i += T::kThreads) {
        const uint32_t qq = i >> 3, e = i & 7;
        if (e < ntail && q0 + qq < a.nq) {
            const float v = a.qprep[size_t(q0 + qq) * dp + tail0 + e];
            sqt[qq * T::kTailStride + e] = L2 ? -v : v;
        }
    }
    const uint32_t ntiles = (r_end - r_begin + T::RB - 1) / T::RB, total = ntiles * nk;
    // Copies the next chunk (kc_next of the row tile at row_next) into stage
    // s_next; rows past the slice repeat its last.
    constexpr uint32_t P = T::KC / 4;
    const uint32_t who = T::kPrivate ? uint32_t(lane) : threadIdx.x;
    const uint32_t my_c = (who % P) * 4, my_r = (T::kPrivate ? uint32_t(wr * RW) : 0u) + who / P;
    uint32_t issued = 0, kc_next = 0, row_next = r_begin + my_r, s_next = 0;
    constexpr uint32_t kStep = (T::kPrivate ? 32 : T::kThreads) / P, kRows = (T::kPrivate ? RW : T::RB) / kStep;
    // The rows of the next tile to copy (a tile ahead, so that a list's entries
    // have arrived when the copies need them).
    uint32_t ids[kRows], ids_next[kRows];
    auto tile_ids = [&](uint32_t row0, uint32_t (&out)[kRows]) {
#pragma unroll
        for (uint32_t i = 0; i < kRows; ++i) out[i] = __ldg(list + min(row0 + i * kStep, r_end - 1));
    };
    if (LIST && total) {
        tile_ids(row_next, ids);
        tile_ids(row_next + T::RB, ids_next);
    }
    auto advance = [&]() {
        if (issued < total) {
            const uint32_t col = kc_next * T::KC + my_c;
            if (col < dp) {
                float* dst = sr + (s_next * T::RB + my_r) * T::kRowStride + my_c;
#pragma unroll
                for (uint32_t i = 0; i < kRows; ++i) {
                    const uint32_t row = LIST ? ids[i] : min(row_next + i * kStep, r_end - 1);
                    cp_async16(dst + i * kStep * T::kRowStride, a.base + size_t(row) * dp + col);
                }
            }
            if (++kc_next == nk) {
                kc_next = 0;
                row_next += T::RB;
                if (LIST) {
#pragma unroll
                    for (uint32_t i = 0; i < kRows; ++i) ids[i] = ids_next[i];
                    tile_ids(row_next + T::RB, ids_next);
                }
            }
            s_next = s_next + 1 == T::kStages ? 0 : s_next + 1;
            ++issued;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < T::kStages - 1; ++s) advance();
    __syncthreads();
    // The pairs this lane finishes: rows 2 my_p, 2 my_p + 1 of query my_q.
    const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4, b3 = lane & 8, b4 = lane & 16;
    const int p0 = (b3 ? 16 : 0) + (b4 ? 8 : 0) + (b2 ? 4 : 0) + (b0 ? 2 : 0) + (b1 ? 1 : 0);
    const int my_q = p0 / RP, my_p = p0 % RP;
    uint32_t thr = 0xFFFFFFFFu;   // bound of my_q
    uint32_t best = 0xFFFFFFFFu;  // smallest admitted distance this lane finished
    const uint32_t mslot = (slice * T::WR + uint32_t(wr)) * RP + uint32_t(my_p);
    const uint32_t nmin = min(nslices * T::WR * RP, kBruteMinima);
    const bool use_minima = a.minima != nullptr && nmin >= kk;
    const uint32_t q = wq0 + uint32_t(my_q);
    const float* qw = sq + wq * QW * T::KC + lane;
    uint32_t stage = 0;
    for (uint32_t tile = 0; tile < ntiles; ++tile) {
        uint64_t acc[NP];  // query i ^ my_q, rows 2j and 2j + 1 at i * RP + j
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[p] = 0ull;
        const float* rw = nullptr;
        for (uint32_t kc = 0; kc < nk; ++kc) {
            asm volatile("cp.async.wait_group %0;" ::"n"(T::kStages - 2) : "memory");
            if (T::kPrivate) __syncwarp();
            else __syncthreads();
            advance();
            rw = sr + (stage * T::RB + wr * RW) * T::kRowStride;
            stage = stage + 1 == T::kStages ? 0 : stage + 1;
            if (!active) continue;
            const float* rk = rw + lane;
            const float* qk = qw + kc * (T::QB * T::KC);
            const float* qp[QW];
#pragma unroll
            for (int i = 0; i < QW; ++i) qp[i] = qk + (i ^ my_q) * T::KC;
            auto step = [&](uint32_t col) {
                uint64_t rv[RP];
#pragma unroll
                for (int j = 0; j < RP; ++j)
                    rv[j] = pack2(rk[2 * j * T::kRowStride + col], rk[(2 * j + 1) * T::kRowStride + col]);
#pragma unroll
                for (int i = 0; i < QW; ++i) {
                    const float x = qp[i][col];
                    const uint64_t xx = pack2(x, x);
#pragma unroll
                    for (int j = 0; j < RP; ++j) acc_pair<L2>(acc[i * RP + j], xx, rv[j]);
                }
            };
            // Full steps of the chunk, then (last chunk) the 8-wide remainder
            // blocks, which go into chain 0 (lanes 0..7).
            const uint32_t k0 = kc * (T::KC / 32), full = 32 * min(uint32_t(T::KC / 32), nfull - min(nfull, k0));
            if (full == T::KC) {
#pragma unroll
                for (uint32_t col = 0; col < T::KC; col += 32) step(col);
            } else {
#pragma unroll 1
                for (uint32_t col = 0; col < full; col += 32) step(col);
                if (lane < 8)
#pragma unroll 1
                    for (uint32_t s = 0; s < rem8; ++s) step(full + 8 * s);
                __syncwarp();
            }
        }
        if (!active) continue;
        const uint32_t shared_thr = q < a.nq ? __ldcg(a.out_count + q) : 0u;
        fold_pairs<32, true>(acc, 8, b3);
        fold_pairs<16, QW == 8>(acc, 16, b4);
        fold_pairs<8, QW == 8>(acc, 4, b2);
        fold_pairs<4, false>(acc, 1, b0);
        fold_pairs<2, false>(acc, 2, b1);
        if (use_minima && tile > 0 && (tile & (tile + 1)) == 0) {
            // Published one tile ago (tile + 1 a power of two).
            constexpr int M = kBruteMinima / 4;
            uint32_t m[M];
            const uint4* src = reinterpret_cast<const uint4*>(a.minima + size_t(min(q, a.nq - 1)) * kBruteMinima);
#pragma unroll
            for (int i = 0; i < M / 4; ++i) {
                const uint4 t4 = __ldcg(src + (lane & 3) * (M / 4) + i);
                m[4 * i] = t4.x;
                m[4 * i + 1] = t4.y;
                m[4 * i + 2] = t4.z;
                m[4 * i + 3] = t4.w;
            }
            thr = min(thr, kth_bound(m, kk, thr));
        }
        const float2 sums = unpack2(acc[0]);
        float s[2] = {sums.x, sums.y};
        const float* rt = rw + 2 * my_p * T::kRowStride + tail0 - (nk - 1) * T::KC;
        const float* qt = sqt + (wq * QW + my_q) * T::kTailStride;
        for (uint32_t e = 0; e < ntail; ++e) {
            const float x = qt[e];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const float y = rt[v * T::kRowStride + e];
                if (L2) {
                    const float d = __fadd_rn(x, y);
                    s[v] = __fadd_rn(s[v], __fmul_rn(d, d));
                } else {
                    s[v] = __fadd_rn(s[v], __fmul_rn(x, y));
                }
            }
        }
        const uint32_t row0 = r_begin + tile * T::RB + uint32_t(wr * RW + 2 * my_p);
        const uint32_t dk0 = fkey(metric_from_sum(a.metric, s[0])), dk1 = fkey(metric_from_sum(a.metric, s[1]));
        thr = min(thr, shared_thr);
        bool want0 = dk0 <= thr && row0 < r_end && q < a.nq;
        bool want1 = dk1 <= thr && row0 + 1 < r_end && q < a.nq;
        if (!LIST && a.filter_bits) {
            want0 = want0 && brute_admits(a, q, row0);
            want1 = want1 && brute_admits(a, q, row0 + 1);
        }
        if (want0) best = min(best, dk0);
        if (want1) best = min(best, dk1);
        if (use_minima && ((tile + 1) & (tile + 2)) == 0 && mslot < kBruteMinima && q < a.nq)
            __stcg(a.minima + size_t(q) * kBruteMinima + mslot, best);
        if (!__any_sync(kFull, want0 || want1)) continue;
#pragma unroll 1
        for (uint32_t v = 0; v < 2; ++v) {
            const bool want = v ? want1 : want0;
            const uint32_t row = LIST && want ? __ldg(list + row0 + v) : row0 + v;
            uint64_t e = (uint64_t(v ? dk1 : dk0) << 32) | row;
            if (want && a.krank) e = (e & 0xFFFFFFFF00000000ull) | __ldg(a.krank + row);
            uint32_t W = __ballot_sync(kFull, want);
            while (W) {
                // The lanes of one query at a time.
                const int src = __ffs(int(W)) - 1;
                const int qi = __shfl_sync(kFull, my_q, src);
                const uint32_t Wi = W & __ballot_sync(kFull, my_q == qi);
                W &= ~Wi;
                TopList t{list_of(warp, qi), wbuf + qi * 32, wmeta[qi].x, wmeta[qi].y};
                const bool merged = top_push(t, Wi, e, kk);
                if (lane == 0) wmeta[qi] = make_uint2(t.n, t.cnt);
                __syncwarp();
                // A merge happened: the list's last entry is a new bound.
                if (merged && t.n == kk) {
                    const uint32_t last = uint32_t(t.L[kk - 1] >> 32);
                    if (my_q == qi) thr = min(thr, last);
                    if (lane == 0) atomicMin(a.out_count + wq0 + qi, last);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (active) {
        for (int i = 0; i < QW; ++i) {
            TopList t{list_of(warp, i), wbuf + i * 32, wmeta[i].x, wmeta[i].y};
            __syncwarp();
            if (t.cnt) top_flush(t, kk);
            if (lane == 0) wmeta[i] = make_uint2(t.n, 0);
            __syncwarp();
        }
    }
    __syncthreads();
    // The lists of the WR warps that share queries become one, written out by
    // the first of them (unused entries ~0).
    if (!active || wr != 0) return;
    for (int i = 0; i < QW; ++i) {
        const uint32_t qg = wq0 + uint32_t(i);
        if (qg >= a.nq) break;
        TopList t{list_of(warp, i), wbuf + i * 32, wmeta[i].x, 0};
        for (int r = 1; r < T::WR; ++r) {
            const int w2 = wq + r * T::WQ;
            const uint64_t* other = list_of(w2, i);
            const uint32_t n2 = meta[w2 * QW + i].x;
            for (uint32_t b = 0; b < n2; b += 32) {
                const uint64_t x = b + uint32_t(lane) < n2 ? other[b + lane] : ~0ull;
                const uint64_t worst = t.n == kk ? t.L[kk - 1] : ~0ull;
                const uint32_t S = __ballot_sync(kFull, x < worst);
                if (S == 0) break;
                batch_merge_gather(t.L, 0, t.n, S, x, kk, t.B);
                __syncwarp();
                t.n = min(t.n + uint32_t(__popc(S)), kk);
            }
        }
        uint64_t* out = a.part + (size_t(qg) * nslices + slice) * kk;
        if (shared_lists) {
            for (uint32_t j = lane; j < kk; j += 32) out[j] = j < t.n ? t.L[j] : ~0ull;
        } else {
            for (uint32_t j = t.n + lane; j < kk; j += 32) out[j] = ~0ull;
        }
    }
}

// Merges the per-slice lists of each query: a block per query, each warp
// taking a share of the entries, filtered by the query's shared bound, into
// a list of its own; warp 0 merges those and writes the results.
constexpr uint32_t kHeads = 4;  // list heads per thread
__global__ void brute_merge_kernel(BruteArgs a, uint32_t kk, uint32_t nslices) {
    extern __shared__ __align__(16) char smem[];
    const uint32_t q = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (a.out_status[q] != 0 || a.k == 0 || a.n == 0) {
        if (threadIdx.x == 0) a.out_count[q] = 0;
        return;
    }
    uint64_t* lists = reinterpret_cast<uint64_t*>(smem);
    uint64_t* bufs = lists + size_t(nw) * kk;
    uint32_t* sizes = reinterpret_cast<uint32_t*>(bufs + size_t(nw) * 32);
    const uint64_t* P = a.part + size_t(q) * nslices * kk;
    const uint64_t n = uint64_t(nslices) * kk;
    // Entries above `bound` cannot be results: the score kernel's shared bound
    // and the kk-th smallest list head.
    uint32_t bound = a.out_count[q];
    if (nslices >= kk && nslices <= blockDim.x * kHeads) {
        uint32_t h[kHeads];
#pragma unroll
        for (uint32_t j = 0; j < kHeads; ++j) {
            const uint32_t s = threadIdx.x + j * blockDim.x;
            h[j] = s < nslices ? uint32_t(__ldcg(P + size_t(s) * kk) >> 32) : 0xFFFFFFFFu;
        }
        uint32_t lo = 0, hi = bound;
        for (int it = 0; it < 24 && hi - lo > 1; ++it) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            uint32_t c = 0;
#pragma unroll
            for (uint32_t j = 0; j < kHeads; ++j)
                if (j * blockDim.x < nslices) c += uint32_t(__syncthreads_count(h[j] <= mid));
            if (c >= kk) hi = mid;
            else lo = mid;
        }
        bound = hi;
    }
    TopList t{lists + size_t(warp) * kk, bufs + warp * 32, 0, 0};
    uint64_t worst = bound == 0xFFFFFFFFu ? ~0ull : (uint64_t(bound) + 1) << 32;  // entries below may be results
    for (uint64_t b0 = uint64_t(warp) * 128; b0 < n; b0 += uint64_t(nw) * 128) {
        uint64_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t i = b0 + uint64_t(32 * j + lane);
            v[j] = i < n ? P[i] : ~0ull;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t W = __ballot_sync(kFull, v[j] < worst);
            if (W == 0) continue;
            top_push(t, W, v[j], kk);
            if (t.n == kk) worst = min(worst, t.L[kk - 1]);
        }
    }
    if (t.cnt) top_flush(t, kk);
    if (lane == 0) sizes[warp] = t.n;
    __syncthreads();  // every thread has read the bound that out_count held
    if (warp != 0) return;
    for (int w2 = 1; w2 < nw; ++w2) {
        const uint64_t* L2p = lists + size_t(w2) * kk;
        const uint32_t n2 = sizes[w2];
        for (uint32_t b = 0; b < n2; b += 32) {
            const uint64_t x = b + uint32_t(lane) < n2 ? L2p[b + lane] : ~0ull;
            const uint32_t S = __ballot_sync(kFull, x < (t.n == kk ? t.L[kk - 1] : ~0ull));
            if (S == 0) break;
            batch_merge_gather(t.L, 0, t.n, S, x, kk, t.B);
            __syncwarp();
            t.n = min(t.n + uint32_t(__popc(S)), kk);
        }
    }
    const uint32_t want = min(t.n, min(a.k, a.n));
    for (uint32_t i = lane; i < want; i += 32) {
        a.out_keys[size_t(q) * a.k + i] = __ldg(a.skeys + uint32_t(t.L[i]));
        a.out_dist[size_t(q) * a.k + i] = kdec(uint32_t(t.L[i] >> 32));
    }
    if (lane == 0) a.out_count[q] = want;
}

// Exact re-rank of tensor-core candidates: every candidate whose approximate
// distance is <= thr2[q] gets its FP32 distance in the reference kernel order;
// a top-k list ordered by (total_cmp distance, key) keeps the best
// (src/brute.rs:131-160). A query whose candidate list overflowed gets status
// 25 and is re-run by the exact FP32 kernels. A block per query: the rows that
// pass are collected 1024 candidates at a time, each warp scores eight of them
// per memory round trip and keeps a list of its own, and warp 0 merges the
// lists. (One warp per query took 346 us for 2000 queries of 768 dimensions
// with 1,250 candidates each, waiting on its row loads 22 of 27 cycles.)
// SMEM_Q: the query in shared memory (left in global memory when it is large).
constexpr uint32_t kRerankBatch = 1024;
template <bool SMEM_Q>
__global__ void __launch_bounds__(256) brute_rerank_kernel(BruteArgs a, const uint64_t* __restrict__ cand,
                                                           const uint32_t* __restrict__ cand_count, uint32_t cand_cap,
                                                           const float* __restrict__ thr2, uint32_t kk) {
    extern __shared__ __align__(16) char smem[];
    __shared__ uint32_t rows[kRerankBatch];
    __shared__ uint32_t nrows, sizes[8];
    const uint32_t q = blockIdx.x, nw = blockDim.x >> 5, warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if (a.out_status[q] != 0) {
        if (threadIdx.x == 0) a.out_count[q] = 0;
        return;
    }
    const uint32_t total = cand_count[q];
    if (total > cand_cap) {
        if (threadIdx.x == 0) a.out_status[q] = 25;
        return;
    }
    float* sq = reinterpret_cast<float*>(smem);
    uint64_t* lists = reinterpret_cast<uint64_t*>(sq + (SMEM_Q ? a.dp : 0));
    uint64_t* bufs = lists + size_t(nw) * kk;
    const float* qv = a.qprep + size_t(q) * a.dp;
    if (SMEM_Q) {
        for (uint32_t i = threadIdx.x * 4; i < a.dp; i += blockDim.x * 4)
            *reinterpret_cast<float4*>(sq + i) = *reinterpret_cast<const float4*>(qv + i);
        qv = sq;
    }
    const float t2 = thr2[q];
    const uint64_t* C = cand + size_t(q) * cand_cap;
    const int g = lane >> 3, g8 = lane & 7;
    TopList t{lists + size_t(warp) * kk, bufs + warp * 32, 0, 0};
    for (uint32_t base = 0; base < total; base += kRerankBatch) {
        __syncthreads();
        if (threadIdx.x == 0) nrows = 0;
        __syncthreads();
        for (uint32_t i = base + threadIdx.x; i < min(total, base + kRerankBatch); i += blockDim.x) {
            const uint64_t c = C[i];
            if (__uint_as_float(uint32_t(c >> 32)) <= t2) rows[atomicAdd(&nrows, 1u)] = uint32_t(c);
        }
        __syncthreads();
        const uint32_t np = nrows;
        for (uint32_t r = warp * 8; r < np; r += nw * 8) {
            const uint32_t sa = r + uint32_t(g), sb = sa + 4;
            const uint32_t ra = rows[min(sa, np - 1)], rb = rows[min(sb, np - 1)];
            const float* xa = a.base + size_t(ra) * a.dp;
            const float* xb = a.base + size_t(rb) * a.dp;
            float d0, d1;
            if (a.metric == 0) group_sum2<true>(xa, xb, qv, int(a.dim), g8, d0, d1);
            else group_sum2<false>(xa, xb, qv, int(a.dim), g8, d0, d1);
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const bool in = g8 == 0 && (h ? sb : sa) < np;
                const uint64_t e = in ? brute_entry(a, metric_from_sum(a.metric, h ? d1 : d0), h ? rb : ra) : ~0ull;
                const uint64_t worst = t.n == kk ? t.L[kk - 1] : ~0ull;
                const uint32_t W = __ballot_sync(kFull, e < worst);
                if (W) top_push(t, W, e, kk);
            }
        }
    }
    if (t.cnt) top_flush(t, kk);
    if (lane == 0) sizes[warp] = t.n;
    __syncthreads();
    if (warp != 0) return;
    for (uint32_t w2 = 1; w2 < nw; ++w2) {
        const uint64_t* other = lists + size_t(w2) * kk;
        const uint32_t n2 = sizes[w2];
        for (uint32_t b = 0; b < n2; b += 32) {
            const uint64_t x = b + uint32_t(lane) < n2 ? other[b + lane] : ~0ull;
            const uint32_t S = __ballot_sync(kFull, x < (t.n == kk ? t.L[kk - 1] : ~0ull));
            if (S == 0) break;
            batch_merge_gather(t.L, 0, t.n, S, x, kk, t.B);
            __syncwarp();
            t.n = min(t.n + uint32_t(__popc(S)), kk);
        }
    }
    const uint32_t want = min(t.n, min(a.k, a.n));
    for (uint32_t i = lane; i < want; i += 32) {
        a.out_keys[size_t(q) * a.k + i] = __ldg(a.skeys + uint32_t(t.L[i]));
        a.out_dist[size_t(q) * a.k + i] = kdec(uint32_t(t.L[i] >> 32));
    }
    if (lane == 0) a.out_count[q] = want;
}

}  // namespace dev

cudaError_t launch_brute_prep(const BruteArgs& a, cudaStream_t stream) {
    dev::brute_prep_kernel<<<(a.nq * 32 + 127) / 128, 128, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_brute_rerank(const BruteArgs& a, const uint64_t* cand, const uint32_t* cand_count, uint32_t cand_cap,
                                const float* thr2, cudaStream_t stream) {
    const uint32_t kk = std::max<uint32_t>(1, std::min<uint32_t>(a.k, a.n ? a.n : 1));
    // Warps per query: eight while the queries do not fill the SMs.
    const uint32_t nw = a.nq >= 1024 ? 4 : 8;
    const bool smem_q = a.dp <= 16384;
    const size_t smem = (smem_q ? size_t(a.dp) * 4 : 0) + size_t(nw) * (kk + 32) * 8;
    auto kern = smem_q ? dev::brute_rerank_kernel<true> : dev::brute_rerank_kernel<false>;
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kern));
    if (e != cudaSuccess) return e;
    kern<<<a.nq, 32 * nw, smem, stream>>>(a, cand, cand_count, cand_cap, thr2, kk);
    return cudaGetLastError();
}

namespace {

// The score kernel's shapes. A warp of eight queries x eight rows is the
// general one. One or two queries take QW = 2 x 32 rows, so that six or seven
// padding queries are not computed and more rows are in flight (one query x
// 200k x 128: 41 us, 57 us with eight queries per warp). Up to eight queries
// put all four warps on rows, up to 16 two: a warp without a query would idle.
using TilePair = dev::BruteTile<2, 32, 1, 4>;
using TileSmall = dev::BruteTile<8, 8, 1, 4>;
using TileMid = dev::BruteTile<8, 8, 2, 2>;
using TileBatch = dev::BruteTile<8, 8, 4, 1>;
using TileLong = dev::BruteTile<8, 8, 1, 1>;  // lists in global memory (k above kSharedListMax)

struct BrutePlan {
    uint32_t qb = 0, rb = 0, threads = 0, slices = 0, kk = 0;
    size_t smem = 0;
    const void* kern = nullptr;  // null: no shape fits
};

constexpr size_t kBruteSmemMax = 227 * 1024;

template <class T, bool LIST>
const void* score_kernel_of(bool l2) {
    return l2 ? reinterpret_cast<const void*>(dev::brute_score_kernel<true, T, LIST>)
              : reinterpret_cast<const void*>(dev::brute_score_kernel<false, T, LIST>);
}

template <class T>
bool take_tile(BrutePlan& p, uint32_t dp, uint32_t list_kk, bool l2, bool rows) {
    const size_t s = T::smem(dp, list_kk);
    if (s > kBruteSmemMax) return false;
    p.qb = T::QB;
    p.rb = T::RB;
    p.threads = T::kThreads;
    p.smem = s;
    p.kern = rows ? score_kernel_of<T, true>(l2) : score_kernel_of<T, false>(l2);
    return true;
}

// Shape and row slices of a batch (`rows`: over a row list); at most
// max_slices lists per query.
cudaError_t plan_brute(uint32_t nq, uint32_t n, uint32_t dp, uint32_t k, int metric, int num_sms, uint32_t max_slices,
                       bool rows, BrutePlan* out) {
    BrutePlan p;
    p.kk = std::max<uint32_t>(1, std::min<uint32_t>(k, n ? n : 1));
    *out = p;
    // Dimensions and k up to 24 rows and 16 lists of k + 1 entries in one
    // block's shared memory are supported.
    if (size_t(24) * dp * 4 + size_t(16) * (p.kk + 1) * 8 > kBruteSmemMax) return cudaErrorInvalidValue;
    const bool l2 = metric == 0;
    bool ok = false;
    if (p.kk <= dev::kSharedListMax) {
        if (nq <= 2) ok = take_tile<TilePair>(p, dp, p.kk, l2, rows);
        if (!ok && nq > 16) ok = take_tile<TileBatch>(p, dp, p.kk, l2, rows);
        if (!ok && nq > 8) ok = take_tile<TileMid>(p, dp, p.kk, l2, rows);
        if (!ok) ok = take_tile<TileSmall>(p, dp, p.kk, l2, rows);
    } else {
        ok = take_tile<TileLong>(p, dp, 0, l2, rows);
    }
    if (!ok) return cudaErrorInvalidValue;
    cudaError_t e = raise_smem_limit(p.kern);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kern, int(p.threads), p.smem);
    if (e != cudaSuccess) return e;
    // Row slices: one full round of resident blocks (several when the query
    // blocks alone come near one), fewer when a slice would fall below one
    // row tile.
    const uint64_t resident = uint64_t(num_sms) * uint64_t(std::max(per_sm, 1));
    const uint64_t qblocks = (nq + p.qb - 1) / p.qb;
    uint64_t s = qblocks >= resident ? (qblocks >= 4 * resident ? 1 : 4 * resident / qblocks) : resident / qblocks;
    s = std::min<uint64_t>(s, (uint64_t(n) + p.rb - 1) / p.rb);
    s = std::min<uint64_t>(std::min<uint64_t>(s, max_slices), 65535);
    p.slices = uint32_t(std::max<uint64_t>(s, 1));
    *out = p;
    return cudaSuccess;
}

int current_sms() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 148;
    return sms;
}

}  // namespace

cudaError_t brute_slices(uint32_t nq, uint32_t n, uint32_t dp, uint32_t k, int metric, uint32_t* slices) {
    BrutePlan p;
    cudaError_t e = plan_brute(nq, n, dp, k, metric, current_sms(), ~0u, false, &p);
    *slices = std::max<uint32_t>(p.slices, 1);
    return e;
}

cudaError_t launch_brute_fp32(const BruteArgs& a, cudaStream_t stream) {
    const bool empty = a.n == 0 || a.k == 0;
    BrutePlan p;
    if (empty) p.kk = p.slices = 1;
    else {
        cudaError_t e = plan_brute(a.nq, a.n, a.dp, a.k, a.metric, current_sms(), a.tiles, a.row_list != nullptr, &p);
        if (e != cudaSuccess) return e;
    }
    dev::brute_prep_kernel<<<(a.nq * 32 + 127) / 128, 128, 0, stream>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (!empty) {
        if (a.row_list) {
            e = cudaMemsetAsync(a.row_list, 0, 4, stream);
            if (e != cudaSuccess) return e;
            dev::brute_rows_kernel<<<(a.n + 255) / 256, 256, 0, stream>>>(a);
            e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
        uint32_t rows_per = ((a.n + p.slices - 1) / p.slices + p.rb - 1) / p.rb * p.rb;
        p.slices = (a.n + rows_per - 1) / rows_per;
        BruteArgs b = a;
        void* argv[] = {&b, &p.kk, &rows_per, &p.slices};
        e = cudaLaunchKernel(p.kern, dim3((a.nq + p.qb - 1) / p.qb, p.slices), dim3(p.threads), argv, p.smem, stream);
        if (e != cudaSuccess) return e;
    }
    // Warps of the merge: about 512 entries each, at most eight.
    const uint64_t entries = uint64_t(p.slices) * p.kk;
    const uint32_t nw = entries >= 4096 ? 8 : (entries >= 1024 ? 4 : (entries >= 512 ? 2 : 1));
    const size_t smem = size_t(nw) * (p.kk + 32) * 8 + nw * 4;
    e = raise_smem_limit(reinterpret_cast<const void*>(dev::brute_merge_kernel));
    if (e != cudaSuccess) return e;
    dev::brute_merge_kernel<<<a.nq, 32 * nw, smem, stream>>>(a, p.kk, p.slices);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Scratch for the allocation-free entry point
// (hnsw_gpu_brute_search_batch_noalloc). The prepared queries and the
// per-slice top-k lists live in this fixed array instead of memory the call
// allocates. Every GPU that loads the library holds it until the process
// exits. Host code must not pass the array's name to a kernel: on the host it
// is only a stand-in, so its device address is looked up once per device.
// ---------------------------------------------------------------------------
namespace {
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices] = {};
}  // namespace

cudaError_t noalloc_scratch_address(void** out) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[device]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[device] = p;
    }
    *out = g_noalloc_ptr[device];
    return cudaSuccess;
}

bool noalloc_layout(uint32_t nq, uint32_t dp, uint32_t kk, uint32_t want_slices, size_t* qprep_bytes,
                    uint32_t* slices) {
    const size_t q = (size_t(nq) * dp * 4 + 255) & ~size_t(255);
    if (q >= kNoAllocScratchBytes) return false;
    const size_t per_slice = size_t(nq) * kk * 8;
    const size_t fit = (kNoAllocScratchBytes - q) / per_slice;
    if (fit < 1) return false;
    *qprep_bytes = q;
    *slices = uint32_t(std::min<size_t>(fit, std::max<uint32_t>(1, want_slices)));
    return true;
}

}  // namespace hnswgpu
