// Team traversal: one block of warps per query, for batches that leave the
// one-warp kernels latency bound (few queries, or filtered walks of very
// uneven length whose longest query is the batch's time).
//
// The walk itself is sequential (HnswIndex::search_layer,
// src/hnsw/search.rs:81-142), but much of it does not depend on its order:
//   fetch   The lists of the best candidates (up to eight) are read and the
//           distances and filter bits of their unvisited neighbors computed
//           into slots in shared memory before the candidates' turn. A
//           neighbor unvisited when its candidate is expanded was unvisited
//           when the list was fetched, so its distance is there.
//   expand  The leading fetched candidates c_0 < c_1 < ... are expanded
//           together as far as the sequential walk would take them in this
//           order: c_i follows if no unvisited neighbor of the ones before it
//           is smaller than c_i, and if the stop rule cannot have fired (with
//           at most A admitted improving neighbors before it, the worst
//           result is at least the one A places below the last). The
//           neighbors that improve on the worst result so far are merged into
//           the results and the candidate queue at once. Neighbors that the
//           sequential walk would have rejected, because an earlier one of the
//           batch had lowered the worst result meanwhile, are at least as far
//           as that worst result: they drop out of the results by rank, and as
//           candidates they can only meet the stop rule. Equal distances
//           (where >= and > differ) are detected, and such a batch's neighbors
//           are taken one by one in list order.
// So the visited set, the expanded nodes and every result are those of the
// one-warp kernels; work is wasted only on fetched candidates that are pushed
// out before their turn.
//
// What bounds it: the latency of one query's chain of steps (a warp alone
// takes about 4.5 cycles per dependent instruction). A warp per query takes
// 6-7,000 cycles per expansion at 50k x 128, ef = 64; fetching ahead with one
// warp expanding candidate by candidate left 3,700 in queue and result
// updates, which is what the joint merge spreads over the block: 3,200 in
// all, of them 1,100 fetching. Per call, a warp per query and a team: one
// query, 50k x 128, ef = 64: 288 and 183 us; 148 queries, 200k x 128, ef =
// 256: 971 and 436 us; 256 requests of the serving mix (30 % filtered, ef to
// 512) on 200k x 128: 19.7 and 7.1 ms; 3,000 filtered int8 queries on 100k x
// 96: 147 and 54 ms. Register caps of 80 and 64 (three and four teams of eight
// warps per SM) were slower: 62 and 79 ms on the last.
//
// Queue: the sorted array C (shared memory, the smallest candidates) and,
// beyond its capacity, an unsorted list in global memory whose entries are
// all above C's; when C runs empty it is refilled with that list's smallest.
// The visited set is a bitmap over node ids, in shared memory when it fits.
#include "traverse.cuh"

namespace hnswgpu {
namespace dev {

constexpr uint32_t kTeamLists = 8;                // candidates expanded together at most
constexpr uint32_t kTeamSlots = 2 * kTeamLists;   // fetched candidates kept
constexpr uint32_t kTeamWarpsMax = 16;
constexpr uint32_t kTeamNew = 96;                 // improving neighbors merged at once
constexpr uint32_t kTeamBins = 1024;              // histogram of a refill

// Block-wide state.
struct TeamCtl {
    uint64_t E[kTeamNew], EA[kTeamNew];     // merged neighbors, and the admitted ones (~0: none)
    uint64_t seq[kTeamNew];                 // the lists' improving neighbors in order, repeats included
    uint32_t seq_adm[kTeamNew];             // whether each is admitted
    uint64_t fmin, fmax;                    // far list: smallest entry; refill window
    uint32_t lmin[kTeamLists];              // per leading candidate: smallest unvisited neighbor (order_key)
    uint32_t lcnt[kTeamLists];              // its improving neighbors, admitted ones << 16
    uint32_t slot_id[kTeamSlots];           // candidate fetched into the slot (kEmpty: none)
    uint32_t slot_adm[kTeamSlots][2];       // admitted neighbors, a mask per 32 list positions (lists up to 64)
    uint32_t fcount, taken, bound_bin;
    uint32_t news;                          // a merge's new entries: for C, for the results << 10, all << 20
    uint64_t sortC[kTeamNew], sortR[kTeamNew];  // in order, and how many old entries are below each
    uint32_t lbC[kTeamNew], lbR[kTeamNew];
    uint32_t rs, head, tail;                // after a refill or a one-by-one merge: results, C[head, tail)
    uint32_t qi, dist0;
    int32_t status, qnorm;
    uint32_t wsum[kTeamWarpsMax];
    float hop[2][32];                       // greedy descent: distances of a list (two hops in turn)
};

// The arrays of a team as offsets into its dynamic shared memory (pointers
// kept in a struct would be read back as generic ones), C and R twice (a
// merge reads one copy and writes the other), and its global arrays.
struct TeamMem {
    uint32_t r_off, r_size, c_off, c_size, ids_off, d_off, hist_off, bm_off, ctl_off;
    uint32_t stride, cap, far_cap, words;
    bool sbm;        // the visited bitmap is in shared memory (else gbm)
    uint64_t* far;
    uint32_t* gbm;
};

__device__ __forceinline__ char* team_smem() {
    extern __shared__ __align__(16) char smem[];
    return smem;
}
__device__ __forceinline__ uint64_t* team_R(const TeamMem& t, uint32_t b) {
    return reinterpret_cast<uint64_t*>(team_smem() + t.r_off + b * t.r_size);
}
__device__ __forceinline__ uint64_t* team_C(const TeamMem& t, uint32_t b) {
    return reinterpret_cast<uint64_t*>(team_smem() + t.c_off + b * t.c_size);
}
__device__ __forceinline__ uint32_t* team_ids(const TeamMem& t) {
    return reinterpret_cast<uint32_t*>(team_smem() + t.ids_off);
}
__device__ __forceinline__ float* team_d(const TeamMem& t) { return reinterpret_cast<float*>(team_smem() + t.d_off); }
__device__ __forceinline__ TeamCtl& team_ctl(const TeamMem& t) {
    return *reinterpret_cast<TeamCtl*>(team_smem() + t.ctl_off);
}

__device__ __forceinline__ bool team_mark(const TeamMem& t, uint32_t id) {
    const uint32_t bit = 1u << (id & 31);
    uint32_t old;
    if (t.sbm) old = atomicOr(reinterpret_cast<uint32_t*>(team_smem() + t.bm_off) + (id >> 5), bit);
    else old = atomicOr(t.gbm + (id >> 5), bit);
    return (old & bit) == 0;
}
__device__ __forceinline__ bool team_seen(const TeamMem& t, uint32_t id) {
    uint32_t word;
    if (t.sbm) word = reinterpret_cast<const uint32_t*>(team_smem() + t.bm_off)[id >> 5];
    else word = __ldcg(t.gbm + (id >> 5));
    return (word >> (id & 31)) & 1u;
}

// The monotone image of a distance with -0 taken as +0: compares as the IEEE
// distances do (never NaN).
__device__ __forceinline__ uint32_t order_key(uint32_t k) { return k == 0x7FFFFFFFu ? 0x80000000u : k; }
__device__ __forceinline__ uint32_t order_key(uint64_t x) { return order_key(uint32_t(x >> 32)); }

// Distances of the neighbors at the list positions in F into out[position].
template <int DK>
__device__ __forceinline__ void team_distances(QueryCtx& c, uint32_t my_id, uint32_t F, float* out) {
    const DeviceIndexView& ix = c.a->ix;
    Ws& w = *c.w;
    const int lane = lane_id(), g = lane >> 3, g8 = lane & 7;
    if constexpr (DK != DK_ANY) {
        chunk_distances<DK>(c, my_id, F);
        if ((F >> lane) & 1u) out[lane] = w.fd[lane];
        __syncwarp();
    } else {
        // int8 codes (the f32 walks are built as DK_L2 and DK_DOT): 16 rows
        // per memory round trip.
        if ((F >> lane) & 1u) w.fr[__popc(F & ((1u << lane) - 1u))] = uint32_t(lane);
        __syncwarp();
        const uint32_t nf = __popc(F);
        const int n16 = int(ix.dc) >> 4;
        for (uint32_t r = 0; r < nf; r += 16) {
            uint32_t id[4], pos[4];
            bool on[4];
            const uint32_t rows = min(nf - r, 16u);  // rows 4 i.. of this round exist iff 4 i < rows
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t at = r + uint32_t(4 * i + g);
                on[i] = at < nf;
                pos[i] = w.fr[on[i] ? at : 0u];
                id[i] = __shfl_sync(kFull, my_id, int(pos[i]));
            }
            int acc[4] = {0, 0, 0, 0}, norm[4] = {0, 0, 0, 0};
            if (c.metric == 0)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (4u * i < rows) norm[i] = __ldg(ix.code_norm + id[i]);
            for (int p = g8; p < n16; p += 8) {
                const int4 y = *(reinterpret_cast<const int4*>(w.qc) + p);
                int4 x[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (4u * i < rows) x[i] = __ldg(reinterpret_cast<const int4*>(ix.codes + size_t(id[i]) * ix.dc) + p);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (4u * i < rows) {
                        acc[i] = __dp4a(x[i].x, y.x, acc[i]);
                        acc[i] = __dp4a(x[i].y, y.y, acc[i]);
                        acc[i] = __dp4a(x[i].z, y.z, acc[i]);
                        acc[i] = __dp4a(x[i].w, y.w, acc[i]);
                    }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (4u * i >= rows) break;
                int v = acc[i];
                v += __shfl_xor_sync(kFull, v, 1, 8);
                v += __shfl_xor_sync(kFull, v, 2, 8);
                v += __shfl_xor_sync(kFull, v, 4, 8);
                const long long l2 = (long long)c.qnorm + (long long)norm[i] - 2ll * (long long)v;
                if (on[i] && g8 == 0) out[pos[i]] = sq_distance(c.metric, v, l2, c.s2);
            }
        }
        __syncwarp();
    }
}

// The fetch phase: this warp's share (the part-th of every `parts` unvisited
// neighbors) of candidate `cid`'s list into slot `s`.
template <int DK>
__device__ __forceinline__ void team_fetch(QueryCtx& c, const TeamMem& t, uint32_t cid, uint32_t s,
                                           uint32_t part, uint32_t parts) {
    const DeviceIndexView& ix = c.a->ix;
    TeamCtl& ctl = team_ctl(t);
#ifdef HNSW_DEVICE_CHECKS
    Ws& w = *c.w;
#endif
    const int lane = lane_id();
    const uint32_t* row = ix.adj0 + size_t(cid) * ix.m0p;
    for (uint32_t base = 0; base < ix.m0; base += 32) {
        uint32_t id = (base + lane < ix.m0) ? __ldg(row + base + lane) : kEmpty;
#ifdef HNSW_DEVICE_CHECKS
        if (!HNSW_CHK(w.chk, id == kEmpty || id < ix.n, 2, id)) id = kEmpty;
#endif
        const bool valid = id != kEmpty;
        const uint32_t V = __ballot_sync(kFull, valid);
        const bool open = valid && !team_seen(t, id);
        const uint32_t O = __ballot_sync(kFull, open);
        const uint32_t rank = __popc(O & ((1u << lane) - 1u));
        const uint32_t F = __ballot_sync(kFull, open && (rank & (parts - 1)) == part);
        if (F) team_distances<DK>(c, id, F, team_d(t) + s * t.stride + base);
        if (part == 0) {
            team_ids(t)[s * t.stride + base + lane] = id;
            const uint32_t A = __ballot_sync(kFull, open && admit(c, id));
            if (lane == 0) ctl.slot_adm[s][base >> 5] = A;
        }
        if (V != kFull) {
            if (part == 0 && base + 32 < ix.m0) team_ids(t)[s * t.stride + base + 32 + lane] = kEmpty;
            break;
        }
    }
    if (part == 0 && lane == 0) ctl.slot_id[s] = cid;
}

// Refills the empty C (copy `b`) from the far list with its smallest entries
// (at least one, at most C's capacity). With ef results, entries worse than
// the worst are dropped first: they can never be expanded. All threads call.
static __device__ __noinline__ void team_refill(TeamMem t, uint32_t b, bool full, uint32_t worst) {
    const int lane = lane_id();
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, nt = blockDim.x;
    TeamCtl& ctl = team_ctl(t);
    uint64_t* const Cb = team_C(t, b);
    uint32_t* const hist = reinterpret_cast<uint32_t*>(team_smem() + t.hist_off);
    __syncthreads();
    if (threadIdx.x == 0) ctl.head = ctl.tail = 0;
    // Compacts the n far entries to those for which keep(x) holds, passing the
    // others to drop(x).
    auto sweep = [&](uint32_t n, auto keep, auto drop) {
        uint32_t kept = 0;
        uint64_t mn = ~0ull, mx = 0;
        for (uint32_t i0 = 0; i0 < n; i0 += nt) {
            const uint32_t i = i0 + threadIdx.x;
            const bool in = i < n;
            const uint64_t x = in ? __ldcg(t.far + i) : 0ull;
            const bool kp = in && keep(x);
            if (in && !kp) drop(x);
            const uint32_t K = __ballot_sync(kFull, kp);
            if (lane == 0) ctl.wsum[warp] = __popc(K);
            __syncthreads();  // every entry of this step is read before any is written
            uint32_t before = 0, all = 0;
            for (uint32_t j = 0; j < warps; ++j) {
                const uint32_t v = ctl.wsum[j];
                before += j < warp ? v : 0u;
                all += v;
            }
            if (kp) {
                __stcg(t.far + kept + before + __popc(K & ((1u << lane) - 1u)), x);
                mn = min(mn, x);
                mx = max(mx, x);
            }
            kept += all;
            __syncthreads();
        }
        mn = warp_min_u64(mn);
        mx = warp_max_u64(mx);
        if (threadIdx.x == 0) {
            ctl.fmin = ~0ull;
            ctl.fmax = 0;
            ctl.fcount = kept;
        }
        __syncthreads();
        if (lane == 0) {
            atomicMin(reinterpret_cast<unsigned long long*>(&ctl.fmin), mn);
            atomicMax(reinterpret_cast<unsigned long long*>(&ctl.fmax), mx);
        }
        __syncthreads();
    };
    if (full) {
        sweep(ctl.fcount, [&](uint64_t x) { return order_key(x) <= worst; }, [](uint64_t) {});
    } else {
        // The window of the selection: smallest and largest entry.
        uint64_t mx = 0;
        for (uint32_t i = threadIdx.x; i < ctl.fcount; i += nt) mx = max(mx, __ldcg(t.far + i));
        mx = warp_max_u64(mx);
        if (threadIdx.x == 0) ctl.fmax = 0;
        __syncthreads();
        if (lane == 0) atomicMax(reinterpret_cast<unsigned long long*>(&ctl.fmax), mx);
        __syncthreads();
    }
    const uint32_t m = ctl.fcount;
    if (m == 0) return;
    uint64_t bound = ~0ull;  // entries below it move to C
    if (m > t.cap) {
        // Radix selection: kTeamBins bins over [lo, lo + 2^bits), `known`
        // entries below the window.
        uint64_t lo = ctl.fmin;
        const uint64_t span = ctl.fmax - lo;
        int bits = span == 0 ? 0 : 64 - __clzll(static_cast<long long>(span));
        uint32_t known = 0;
        for (int pass = 0; pass < 7; ++pass) {
            const int sh = max(bits - 10, 0);
            for (uint32_t i = threadIdx.x; i < kTeamBins; i += nt) hist[i] = 0;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < m; i += nt) {
                const uint64_t x = __ldcg(t.far + i);
                const uint64_t off = x - lo;
                if (x >= lo && (bits >= 64 || (off >> bits) == 0)) atomicAdd(&hist[uint32_t(off >> sh)], 1u);
            }
            __syncthreads();
            if (warp == 0) {
                // Largest bin count j with known + (entries in bins below j) <= cap.
                uint32_t sum = 0;
                for (uint32_t i = 0; i < kTeamBins / 32; ++i) sum += hist[lane * (kTeamBins / 32) + i];
                uint32_t incl = sum;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t o = __shfl_up_sync(kFull, incl, off);
                    if (lane >= off) incl += o;
                }
                uint32_t at = known + incl - sum, j = lane * (kTeamBins / 32), taken = at;
                bool open = at <= t.cap;
                for (uint32_t i = 0; i < kTeamBins / 32 && open; ++i) {
                    at += hist[lane * (kTeamBins / 32) + i];
                    open = at <= t.cap;
                    if (open) {
                        ++j;
                        taken = at;
                    }
                }
                // The last lane whose range begins within the cap decides.
                const uint32_t L = __ballot_sync(kFull, known + incl - sum <= t.cap);
                const int last = 31 - __clz(int(L));
                const uint32_t jj = __shfl_sync(kFull, j, last), tt = __shfl_sync(kFull, taken, last);
                if (lane == 0) {
                    ctl.bound_bin = jj;
                    ctl.taken = tt;
                }
            }
            __syncthreads();
            const uint32_t j = ctl.bound_bin, taken = ctl.taken;
            __syncthreads();
            bound = lo + (uint64_t(j) << sh);
            if (2 * taken >= t.cap || sh == 0) break;
            // Too few below the boundary bin: split it.
            known = taken;
            lo = bound;
            bits = sh;
        }
    }
    // Move the entries below the bound to C and sort them.
    if (threadIdx.x == 0) ctl.taken = 0;
    __syncthreads();
    const uint32_t n0 = ctl.fcount;
    if (bound == ~0ull) {
        for (uint32_t i = threadIdx.x; i < n0; i += nt) Cb[i] = __ldcg(t.far + i);
        __syncthreads();
        if (threadIdx.x == 0) {
            ctl.taken = n0;
            ctl.fcount = 0;
            ctl.fmin = ~0ull;
        }
        __syncthreads();
    } else {
        sweep(n0, [&](uint64_t x) { return x >= bound; }, [&](uint64_t x) { Cb[atomicAdd(&ctl.taken, 1u)] = x; });
    }
    const uint32_t got = ctl.taken;
    uint32_t p2 = 32;
    while (p2 < got) p2 <<= 1;
    uint64_t* A = Cb;
    for (uint32_t i = got + threadIdx.x; i < p2; i += nt) A[i] = ~0ull;
    __syncthreads();
    for (uint32_t size = 2; size <= p2; size <<= 1)
        for (uint32_t half = size >> 1; half > 0; half >>= 1) {
            for (uint32_t i = threadIdx.x; i < p2 / 2; i += nt) {
                const uint32_t lo = 2 * i - (i & (half - 1)), hi = lo + half;
                const uint64_t x = A[lo], y = A[hi];
                const bool up = (lo & size) == 0;
                if ((x > y) == up) {
                    A[lo] = y;
                    A[hi] = x;
                }
            }
            __syncthreads();
        }
    if (threadIdx.x == 0) {
        ctl.head = 0;
        ctl.tail = got;
    }
    __syncthreads();
}

// One query by the block. Returns its status (ST_OVERFLOW: the retry pass).
template <int DK>
__device__ __forceinline__ int32_t team_query(const SearchArgs& a, Ws& w, const TeamMem& t, uint32_t qi) {
    const DeviceIndexView& ix = a.ix;
    const int lane = lane_id();
    const uint32_t tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, warps = nt >> 5;
    TeamCtl& ctl = team_ctl(t);
    QueryCtx c;
    c.a = &a;
    c.w = &w;
    c.qi = qi;
    c.metric = ix.metric;
    c.quant = DK == DK_ANY && a.quantized != 0 && ix.quantized != 0;
    c.s2 = __fmul_rn(ix.scale, ix.scale);
    c.qnorm = 0;
    c.use_filter = a.filter_bits != nullptr && (a.filter_used == nullptr || a.filter_used[qi] != 0);
    const size_t fsel = a.filter_ids ? size_t(a.filter_ids[qi]) : size_t(qi);
    c.fbits = a.filter_bits + (a.filter_stride ? fsel * a.filter_stride : 0);
    c.fnbits = a.filter_nbits;
    c.by_node = a.filter_by_node != 0;
    const uint32_t k = min(a.ks ? a.ks[qi] : a.k, a.out_stride);
    uint32_t ef = a.efs ? a.efs[qi] : a.ef;
    // Query by warp 0, the visited set cleared by all.
    if (warp == 0) {
        int32_t st = prepare(c, a.queries + size_t(qi) * ix.dim);
        if (st == ST_OK && a.quantized && !ix.quantized) st = ST_QDISABLED;
        if (lane == 0) {
            ctl.status = st;
            ctl.qnorm = c.qnorm;
            ctl.dist0 = 0;
            ctl.fcount = 0;
            ctl.fmin = ~0ull;
        }
    }
    {
        const uint4 z = make_uint4(0, 0, 0, 0);
        if (t.sbm) {
            uint4* b4 = reinterpret_cast<uint4*>(team_smem() + t.bm_off);
            for (uint32_t i = tid; i < (t.words >> 2); i += nt) b4[i] = z;
        } else {
            uint4* b4 = reinterpret_cast<uint4*>(t.gbm);
            for (uint32_t i = tid; i < (t.words >> 2); i += nt) b4[i] = z;
            __threadfence();
        }
    }
    if (tid < kTeamSlots) ctl.slot_id[tid] = kEmpty;
    __syncthreads();
    int32_t st = ctl.status;
    c.qnorm = ctl.qnorm;
    uint32_t count = 0;
    if (st == ST_OK && k != 0 && ix.live != 0 && ix.entry != kEmpty) {
        ef = max(ef, k);
        if (ef > w.ef_cap) return ST_OVERFLOW;
        const float d0 = group_distance<DK>(c, ix.entry, lane & 7);
        c.cnt.dist_up++;
        uint64_t ep = pack(d0, ix.entry);
        // greedy_closest (src/hnsw/search.rs:49-68): each warp computes a
        // share of the list's distances, all warps take the same minimum.
        const uint32_t share = warps == 16 ? 0x00010001u : (warps == 8 ? 0x01010101u : 0x11111111u);
        uint32_t hop = 0;
        for (uint32_t layer = ix.top; layer >= 1; --layer) {
            for (;;) {
                const uint32_t from = pid(ep);
#ifdef HNSW_DEVICE_CHECKS
                if (!HNSW_CHK(w.chk, from < ix.n, 4, from)) break;
#endif
                const uint32_t* blk = ix.adjU + size_t(__ldg(ix.up_off + from) + (layer - 1)) * ix.mp;
                c.cnt.exp_up++;
                float bd = pdist(ep);
                uint32_t bid = from;
                for (uint32_t base = 0; base < ix.m; base += 32) {
                    uint32_t id = (base + lane < ix.m) ? __ldg(blk + base + lane) : kEmpty;
#ifdef HNSW_DEVICE_CHECKS
                    if (!HNSW_CHK(w.chk, id == kEmpty || id < ix.n, 2, id)) id = kEmpty;
#endif
                    const uint32_t V = __ballot_sync(kFull, id != kEmpty);
                    if (V == 0) break;
                    const uint32_t F = V & (share << warp);
                    float* hd = ctl.hop[hop & 1];
                    ++hop;
                    if (F) team_distances<DK>(c, id, F, hd);
                    __syncthreads();
                    c.cnt.dist_up += __popc(V);
                    float d = ((V >> lane) & 1u) ? hd[lane] : __int_as_float(0x7f800000);
                    int idx = lane;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) {
                        const float od = __shfl_down_sync(kFull, d, off);
                        const int oi = __shfl_down_sync(kFull, idx, off);
                        if (od < d || (od == d && oi < idx)) {
                            d = od;
                            idx = oi;
                        }
                    }
                    d = __shfl_sync(kFull, d, 0);
                    idx = __shfl_sync(kFull, idx, 0);
                    if (((V >> idx) & 1u) && d < bd) {
                        bd = d;
                        bid = __shfl_sync(kFull, id, idx);
                    }
                    if (V != kFull) break;
                }
                if (bid == from) break;
                ep = (uint64_t(fkey(bd)) << 32) | bid;
            }
        }
        // Layer 0.
        const bool adm0 = admit(c, pid(ep));
        uint32_t b = 0;  // the live copy of R and C
        uint32_t rs = adm0 ? 1u : 0u, head = 0, tail = 1;
        if (tid == 0) {
            team_mark(t, pid(ep));
            team_C(t, 0)[0] = ep;
            if (adm0) team_R(t, 0)[0] = ep;
            ctl.news = 0;
        }
        uint32_t fresh_seen = 0;
        bool fail = false;
        __syncthreads();
        for (;;) {
            const uint64_t* R = team_R(t, b);
            const uint64_t* C = team_C(t, b) + head;
            const uint32_t nc = tail - head;
            const bool rfull = rs >= ef;
            const uint32_t worst = rfull ? order_key(R[rs - 1]) : 0xFFFFFFFFu;
            if (nc == 0) {
                if (ctl.fcount == 0) break;
                team_refill(t, b, rfull, worst);
                head = ctl.head;
                tail = ctl.tail;
                __syncthreads();
                if (tail == head) break;
                continue;
            }
            // The leading candidates and their slots (lane i of every warp
            // holds candidate i's).
            const uint32_t lists = min(min(nc, kTeamLists), warps);
            const uint64_t lc = uint32_t(lane) < lists ? C[lane] : ~0ull;
            const uint32_t sid = ctl.slot_id[lane & (kTeamSlots - 1)];
            uint32_t found = 0;
#pragma unroll
            for (int i = 0; i < int(kTeamLists); ++i) {
                const uint32_t m = __ballot_sync(kFull, sid == __shfl_sync(kFull, pid(lc), i));
                if (lane == i) found = m & ((1u << kTeamSlots) - 1u);
            }
            const bool have = uint32_t(lane) < lists;
            if (!have) found = 0;
            const uint32_t cached = __ballot_sync(kFull, found != 0);
            if (rfull && order_key(__shfl_sync(kFull, uint32_t(lc >> 32), 0)) > worst) break;
            if (!(cached & 1u)) {
                // Fetch the leading candidates that have no slot (every warp has
                // read the slots' ids before one is written).
                __syncthreads();
                const uint32_t U = ~cached & ((1u << lists) - 1u);
                const uint32_t used = __reduce_or_sync(kFull, found);
                const uint32_t jobs = __popc(U);
                const uint32_t span = jobs <= 1 ? 1u : (jobs <= 2 ? 2u : (jobs <= 4 ? 4u : 8u));
                const uint32_t parts = max(warps / span, 1u);
                const uint32_t job = warp / parts;
                if (job < jobs) {
                    const uint32_t cid = __shfl_sync(kFull, pid(lc), nth_set(U, int(job)));
                    const uint32_t s = uint32_t(nth_set(~used & ((1u << kTeamSlots) - 1u), int(job)));
#ifdef HNSW_DEVICE_CHECKS
                    if (HNSW_CHK(w.chk, cid < ix.n, 3, cid))
#endif
                        team_fetch<DK>(c, t, cid, s, warp & (parts - 1), parts);
                }
                // The next lists into L1.
                if (warp < kTeamLists && lane == 0 && warp + lists < nc)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(ix.adj0 + size_t(pid(C[warp + lists])) * ix.m0p));
                __syncthreads();
                continue;
            }
            // Warp i looks at the i-th: its unvisited neighbors, those that
            // improve on the worst result and the admitted ones of them.
            uint32_t my_id[2] = {kEmpty, kEmpty}, open[2] = {0, 0}, imp[2] = {0, 0}, adm[2] = {0, 0}, slot = 0;
            float my_d[2] = {0.0f, 0.0f};
            if (warp < lists && ((cached >> warp) & 1u)) {
                slot = uint32_t(__ffs(int(__shfl_sync(kFull, found, int(warp)))) - 1);
                uint32_t mn = 0xFFFFFFFFu;
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    if (32 * h >= ix.m0) break;
                    my_id[h] = team_ids(t)[slot * t.stride + 32 * h + lane];
                    const bool valid = my_id[h] != kEmpty;
                    const bool o = valid && !team_seen(t, my_id[h]);
                    my_d[h] = team_d(t)[slot * t.stride + 32 * h + lane];
                    const uint32_t kd = o ? order_key(fkey(my_d[h])) : 0xFFFFFFFFu;
                    open[h] = __ballot_sync(kFull, o);
                    imp[h] = __ballot_sync(kFull, o && (!rfull || kd < worst));
                    adm[h] = imp[h] & ctl.slot_adm[slot][h];
                    mn = min(mn, kd);
                    if (__ballot_sync(kFull, valid) != kFull) break;
                }
                mn = __reduce_min_sync(kFull, mn);
                if (lane == 0) {
                    ctl.lmin[warp] = mn;
                    ctl.lcnt[warp] = (__popc(imp[0]) + __popc(imp[1])) | ((__popc(adm[0]) + __popc(adm[1])) << 16);
                }
            }
            __syncthreads();
            // How many of them the sequential walk takes in this order (every
            // warp decides the same; lane i holds candidate i).
            const bool on = have && found != 0;
            uint32_t pm = on ? ctl.lmin[lane & (kTeamLists - 1)] : 0xFFFFFFFFu;  // inclusive prefix minimum
            const uint32_t own = on ? ctl.lcnt[lane & (kTeamLists - 1)] : 0u;
            uint32_t sums = own;                                               // inclusive prefix sums
#pragma unroll
            for (int off = 1; off < int(kTeamLists); off <<= 1) {
                const uint32_t om = __shfl_up_sync(kFull, pm, off), os = __shfl_up_sync(kFull, sums, off);
                if (lane >= off) {
                    pm = min(pm, om);
                    sums += os;
                }
            }
            const uint32_t prev_min = __shfl_up_sync(kFull, pm, 1);
            const uint32_t A = (sums - own) >> 16;  // admitted improving neighbors before this candidate, at most
            const uint32_t lk = order_key(lc);
            bool ok = on;
            if (ok && lane > 0) {
                ok = lk < prev_min && (sums & 0xFFFFu) <= kTeamNew;
                if (rs + A >= ef) ok = ok && A < ef && lk <= order_key(R[ef - 1 - A]);
            }
            const uint32_t j = uint32_t(__ffs(int(~__ballot_sync(kFull, ok))) - 1);
            // Expand candidates 0..j-1: mark their neighbors, list the
            // improving ones in list order (holes for those another list of
            // the batch has marked first).
            const uint32_t ne = __shfl_sync(kFull, sums, int(j) - 1) & 0xFFFFu;
            const uint32_t fcount = ctl.fcount;
            const uint64_t fmin = fcount ? ctl.fmin : ~0ull;  // entries above it go to the far list
            uint32_t at = __shfl_sync(kFull, sums - own, int(warp) & 31) & 0xFFFFu;
            if (warp < j) {
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    if (open[h] == 0) continue;
                    const bool fresh = ((open[h] >> lane) & 1u) && team_mark(t, my_id[h]);
                    fresh_seen += __popc(__ballot_sync(kFull, fresh));
                    if (imp[h] == 0) continue;
                    const uint64_t x = pack(my_d[h], my_id[h]);
                    const bool in = (imp[h] >> lane) & 1u, inA = (adm[h] >> lane) & 1u;
                    if (in) {
                        const uint32_t e = at + __popc(imp[h] & ((1u << lane) - 1u));
                        ctl.E[e] = fresh ? x : ~0ull;
                        ctl.EA[e] = fresh && inA ? x : ~0ull;
                        ctl.seq[e] = x;
                        ctl.seq_adm[e] = inA ? 1u : 0u;
                    }
                    at += __popc(imp[h]);
                    const uint32_t nC = __popc(__ballot_sync(kFull, in && fresh && x <= fmin));
                    const uint32_t nR = __popc(__ballot_sync(kFull, inA && fresh));
                    const uint32_t nF = __popc(__ballot_sync(kFull, in && fresh));
                    if (lane == 0) atomicAdd(&ctl.news, nC | (nR << 10) | (nF << 20));
                }
                if (lane == 0) ctl.slot_id[slot] = kEmpty;
            }
            c.cnt.exp0 += j;
            __syncthreads();
            head += j;
            if (ne == 0) continue;
            // Merge, first the new entries: sort them by rank and find their
            // places in C and in the results (a warp of its own for each).
            const uint64_t* Cj = team_C(t, b) + head;
            const uint32_t ncj = nc - j;
            const uint32_t news = ctl.news, new_c = news & 1023u, new_r = (news >> 10) & 1023u, new_all = news >> 20;
            const uint32_t nep = (ne + 31u) & ~31u;
            uint32_t tie = 0;  // largest key of a new entry with an equal among the new ones or the results
            for (uint32_t it = tid; it < 2 * nep; it += nt) {
                const bool toC = it < nep;
                const uint32_t i = toC ? it : it - nep;
                if (i >= ne) continue;
                const uint64_t v = ctl.E[i];
                if (v == ~0ull) continue;
                const uint64_t* L = toC ? ctl.E : ctl.EA;
                uint32_t rank = 0;
#pragma unroll 4
                for (uint32_t e = 0; e < ne; ++e) rank += L[e] < v ? 1u : 0u;
                const uint64_t* S = toC ? Cj : R;
                const uint32_t sn = toC ? ncj : rs;
                const uint32_t lb = lower_bound(S, 0, sn, v);
                if (toC) {
                    ctl.sortC[rank] = v;
                    ctl.lbC[rank] = lb;
                } else {
                    const uint32_t kv = order_key(v);
                    if ((lb < sn && order_key(S[lb]) == kv) || (lb > 0 && order_key(S[lb - 1]) == kv)) tie = max(tie, kv);
                    if (ctl.EA[i] != ~0ull) {
                        ctl.sortR[rank] = v;
                        ctl.lbR[rank] = lb;
                    }
                }
            }
            __syncthreads();
            // Then every entry to its place in the other copy: an old one moves
            // up by the new ones placed at or before it. C keeps its `cap`
            // smallest; the rest, and new entries above the far list's minimum,
            // join the far list (dropped when they are worse than the worst of
            // ef results).
            uint64_t* R2 = team_R(t, b ^ 1);
            uint64_t* C2 = team_C(t, b ^ 1);
            auto to_far = [&](uint64_t v) {
                if (order_key(v) > worst) return;
                const uint32_t f = atomicAdd(&ctl.fcount, 1u);
                if (f < t.far_cap) __stcg(t.far + f, v);
                atomicMin(reinterpret_cast<unsigned long long*>(&ctl.fmin), static_cast<unsigned long long>(v));
            };
            // (Each kind of item starts on a warp of its own.)
            const uint32_t nall = (new_all + 31u) & ~31u, nrp = (new_r + 31u) & ~31u, rsp = (rs + 31u) & ~31u;
            const uint32_t items = nall + nrp + rsp + ncj;
            for (uint32_t it = tid; it < items; it += nt) {
                uint32_t i = it;
                if (i < nall) {
                    if (i >= new_all) continue;
                    const uint64_t v = ctl.sortC[i];
                    const uint32_t pos = ctl.lbC[i] + i;
                    if (pos < t.cap && v <= fmin) C2[pos] = v;
                    else to_far(v);
                    if (i + 1 < new_all && order_key(v) == order_key(ctl.sortC[i + 1])) tie = max(tie, order_key(v));
                    continue;
                }
                i -= nall;
                if (i < nrp) {
                    if (i >= new_r) continue;
                    const uint32_t pos = ctl.lbR[i] + i;
                    if (pos < ef) R2[pos] = ctl.sortR[i];
                    continue;
                }
                i -= nrp;
                if (i < rsp) {
                    if (i >= rs) continue;
                    const uint64_t v = R[i];
                    uint32_t pos = i;
#pragma unroll 4
                    for (uint32_t e = 0; e < new_r; ++e) pos += ctl.lbR[e] <= i ? 1u : 0u;
                    if (pos < ef) R2[pos] = v;
                    continue;
                }
                i -= rsp;
                const uint64_t v = Cj[i];
                uint32_t pos = i;
#pragma unroll 4
                for (uint32_t e = 0; e < new_c; ++e) pos += ctl.lbC[e] <= i ? 1u : 0u;
                if (pos < t.cap) C2[pos] = v;
                else to_far(v);
            }
            // A tie matters only at the worst result: the sequential walk
            // compares a neighbor with it, and it never falls below the merge's.
            bool one_by_one = __syncthreads_or(tie != 0);
            if (one_by_one)
                one_by_one = __syncthreads_or(rs + new_r >= ef && tie != 0 && tie >= order_key(R2[ef - 1]));
            if (one_by_one) {
                // Warp 0 takes the new entries one by one on the old copies
                // (the far list as it was), each where the lists have it
                // first: of lists that share a neighbor, any may have marked it.
                if (warp == 0) {
                    uint64_t* Cw = team_C(t, b);
                    uint64_t* Rw = team_R(t, b);
                    uint32_t tl = ncj, r = rs, fc = fcount;
                    uint64_t fm = fcount ? fmin : ~0ull;
                    // C's live range moves to its start first: these merges
                    // do not reset `head`, so many in a row would run the
                    // range out of the array, down to an empty one at its end.
                    if (head > 0)
                        for (uint32_t i0 = 0; i0 < ncj; i0 += 32) {
                            const uint32_t i = i0 + uint32_t(lane);
                            const uint64_t v = i < ncj ? Cw[head + i] : 0ull;
                            __syncwarp();
                            if (i < ncj) Cw[i] = v;
                            __syncwarp();
                        }
                    for (uint32_t e = 0; e < ne; ++e) {
                        const uint64_t x = ctl.seq[e];
                        bool repeat = false;
                        for (uint32_t f = lane; f < e; f += 32) repeat |= ctl.seq[f] == x;
                        if (__any_sync(kFull, repeat)) continue;
                        if (r >= ef && !(pdist(x) < pdist(Rw[r - 1]))) continue;
                        uint64_t to_far = ~0ull;
                        if (fc && x > fm) {
                            to_far = x;
                        } else if (tl >= t.cap) {
                            to_far = Cw[tl - 1];  // the largest leaves C
                            __syncwarp();
                            if (x > to_far) {
                                to_far = x;
                            } else {
                                sorted_insert(Cw, 0, tl - 1, x);
                            }
                        } else {
                            sorted_insert(Cw, 0, tl, x);
                            ++tl;
                        }
                        if (to_far != ~0ull) {
                            if (lane == 0 && fc < t.far_cap) __stcg(t.far + fc, to_far);
                            ++fc;
                            fm = min(fm, to_far);
                        }
                        if (ctl.seq_adm[e]) {
                            sorted_insert(Rw, 0, r, x);
                            r = min(r + 1, ef);
                        }
                        __syncwarp();
                    }
                    if (lane == 0) {
                        ctl.tail = tl;
                        ctl.rs = r;
                        ctl.fcount = fc;
                        ctl.fmin = fm;
                    }
                }
                __syncthreads();
                head = 0;
                tail = ctl.tail;
                rs = ctl.rs;
            } else {
                b ^= 1;
                head = 0;
                tail = min(ncj + new_c, t.cap);
                rs = min(rs + new_r, ef);
            }
            if (tid == 0) ctl.news = 0;
            if (ctl.fcount > t.far_cap) {
                fail = true;
                break;
            }
        }
        __syncthreads();
        if (fail) return ST_OVERFLOW;
        if (a.counters && lane == 0) atomicAdd(&ctl.dist0, fresh_seen);
        const uint32_t n = rs;
        count = min(n, k);
        uint64_t* Rf = team_R(t, b);
        uint64_t* key_of = team_R(t, b ^ 1);
        if (c.quant) {
            // Exact distances for the survivors (src/hnsw/mod.rs:494-498).
            uint64_t* X = team_R(t, b ^ 1);
            for (uint32_t r = warp * 4; r < n; r += warps * 4) {
                const uint32_t i = r + uint32_t(lane >> 3);
                const uint32_t id = pid(Rf[i < n ? i : 0]);
                const float d = group_exact(c, id, lane & 7);
                if (i < n && (lane & 7) == 0) X[i] = pack(d, id);
            }
            __syncthreads();
            key_of = Rf;
            Rf = X;
        }
        for (uint32_t i = tid; i < n; i += nt)
            key_of[i] = ix.keys_are_ids ? uint64_t(pid(Rf[i])) : __ldg(ix.keys + pid(Rf[i]));
        __syncthreads();
        // Sort by (total_cmp distance, key) and keep k (src/hnsw/mod.rs:501-510).
        // The f32 walk's results are sorted by (distance, id) already.
        for (uint32_t i = tid; i < n; i += nt) {
            const uint32_t dk = uint32_t(Rf[i] >> 32);
            const uint64_t key = key_of[i];
            uint32_t rank = 0;
            if (c.quant) {
                for (uint32_t o = 0; o < n; ++o) {
                    const uint32_t ok = uint32_t(Rf[o] >> 32);
                    rank += (ok < dk || (ok == dk && key_of[o] < key)) ? 1u : 0u;
                }
            } else {
                rank = i;
                for (uint32_t o = i; o > 0 && uint32_t(Rf[o - 1] >> 32) == dk; --o) rank -= key_of[o - 1] > key ? 1u : 0u;
                for (uint32_t o = i + 1; o < n && uint32_t(Rf[o] >> 32) == dk; ++o) rank += key_of[o] < key ? 1u : 0u;
            }
            if (rank < k) {
                const size_t o = size_t(qi) * a.out_stride + rank;
                a.out_keys[o] = key;
                a.out_dist[o] = kdec(dk);
            }
        }
    }
    if (a.publish) __threadfence_system();
    __syncthreads();
    if (tid == 0) {
        a.out_count[qi] = st == ST_OK ? count : 0u;
        if (a.publish) __threadfence_system();
        a.out_status[qi] = st;
        if (a.counters) {
            a.counters[4 * size_t(qi) + 0] = ctl.dist0;
            a.counters[4 * size_t(qi) + 1] = c.cnt.exp0;
            a.counters[4 * size_t(qi) + 2] = c.cnt.dist_up;
            a.counters[4 * size_t(qi) + 3] = c.cnt.exp_up;
        }
    }
    return st;
}

// Shared-memory layout of a team; returns its size.
__host__ __device__ inline size_t team_layout(uint32_t dp, uint32_t dc, uint32_t m0p, const TeamGeometry& g,
                                              size_t (&off)[8]) {
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o = align_up(o + bytes, 16);
        return at;
    };
    // C is sorted as a power of two of entries when it is refilled.
    off[0] = take(size_t(dp) * 4);
    off[1] = take(dc);
    off[2] = take(size_t(g.ef_cap + 1) * 16);
    off[3] = take(size_t(g.cand_cap + 32) * 16);
    off[4] = take(size_t(g.warps) * 256 + kTeamBins * 4);
    off[5] = take(size_t(kTeamSlots) * m0p * 8);
    off[6] = take(sizeof(TeamCtl));
    off[7] = take(size_t(g.bitmap_words) * 4);
    return o;
}

template <int DK>
__global__ void __launch_bounds__(512, 1) search_team_kernel(SearchArgs a, TeamGeometry g) {
    if (a.route && *a.route != kRouteTeam) return;
    char* smem = team_smem();
    const DeviceIndexView& ix = a.ix;
    const uint32_t warp = threadIdx.x >> 5;
    size_t off[8];
    team_layout(ix.dp, ix.dc, ix.m0p, g, off);
    TeamMem t;
    t.r_off = uint32_t(off[2]);
    t.r_size = (g.ef_cap + 1) * 8;
    t.c_off = uint32_t(off[3]);
    t.c_size = (g.cand_cap + 32) * 8;
    t.hist_off = uint32_t(off[4]);
    t.ids_off = uint32_t(off[5]);
    t.d_off = uint32_t(off[5]) + kTeamSlots * ix.m0p * 4;
    t.ctl_off = uint32_t(off[6]);
    t.bm_off = uint32_t(off[7]);
    t.sbm = g.bitmap_words != 0;
    t.words = g.bitmap_words ? g.bitmap_words : a.spill_words;
    t.gbm = a.spill_bits + size_t(blockIdx.x) * a.spill_words;
    t.stride = ix.m0p;
    t.cap = g.cand_cap;
    t.far = a.team_far + size_t(blockIdx.x) * g.far_cap;
    t.far_cap = g.far_cap;
    Ws w;
    w.qf = reinterpret_cast<float*>(smem + off[0]);
    w.qc = reinterpret_cast<int8_t*>(smem + off[1]);
    w.qt = nullptr;
    w.fr = reinterpret_cast<uint32_t*>(smem + off[4] + kTeamBins * 4 + warp * 256);
    w.fd = reinterpret_cast<float*>(w.fr + 32);
    w.stage = nullptr;
    w.stage_rows = w.stage_row_bytes = 0;
    w.fi = nullptr;
    w.fnorm = nullptr;
    w.ef_cap = g.ef_cap;
#ifdef HNSW_DEVICE_CHECKS
    w.chk = a.chk;
#endif
    TeamCtl& ctl = team_ctl(t);
    const uint32_t queries = a.team_count ? *a.team_count : a.nq;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) ctl.qi = atomicAdd(a.work_next, 1u);
        __syncthreads();
        uint32_t qi = ctl.qi;
        if (qi >= queries) break;
        if (a.order) qi = a.order[qi];
        const int32_t st = team_query<DK>(a, w, t, qi);
        if (st == ST_OVERFLOW && threadIdx.x == 0) {
            a.overflow_list[atomicAdd(a.overflow_count, 1u)] = qi;
            a.out_status[qi] = ST_OVERFLOW;
        }
    }
}

// Expected expansions of a query: a filtered walk goes on until ef admitted
// nodes are found, i.e. about ef / selectivity (the index's size at most). The
// selectivity is that of 32 words spread over the nodes where bits are indexed
// by node, else of 256 nodes' keys: keys need not lie in [0, n).
__device__ __forceinline__ float expected_work(const SearchArgs& a, uint32_t qi) {
    const DeviceIndexView& ix = a.ix;
    const uint32_t k = min(a.ks ? a.ks[qi] : a.k, a.out_stride);
    float cost = float(max(a.efs ? a.efs[qi] : a.ef, k));
    if (a.filter_bits != nullptr && (a.filter_used == nullptr || a.filter_used[qi] != 0)) {
        const size_t fsel = a.filter_ids ? size_t(a.filter_ids[qi]) : size_t(qi);
        const uint64_t* bits = a.filter_bits + (a.filter_stride ? fsel * a.filter_stride : 0);
        uint32_t set = 0, of = 0;
        if (ix.keys_are_ids || a.filter_by_node) {
            const uint32_t nwords = max(ix.n >> 6, 1u), m = min(nwords, 32u);
            of = 64u * m;
#pragma unroll 8
            for (uint32_t i = 0; i < m; ++i) {
                const uint64_t w = nwords > 32u ? (uint64_t(nwords) * i) >> 5 : i;
                if (w * 64 < a.filter_nbits) set += uint32_t(__popcll(static_cast<long long>(__ldg(bits + w))));
            }
        } else {
            of = min(ix.n, 256u);
#pragma unroll 8
            for (uint32_t i = 0; i < of; ++i) {
                const uint64_t key = __ldg(ix.keys + (ix.n > 256u ? (uint64_t(ix.n) * i) >> 8 : i));
                if (key < a.filter_nbits) set += uint32_t(__ldg(bits + (key >> 6)) >> (key & 63)) & 1u;
            }
        }
        cost = cost * float(max(of, 1u)) / float(max(set, 1u));
    }
    return fminf(fmaxf(cost, 1.0f), float(max(ix.live, 1u)));
}

// Queries in descending order of expected work, so that the longest walks
// start first (buckets of a quarter octave, any order inside one), and the
// route of the batch: a warp or a team per query. One block.
//
// The route compares the two kernels' expected times: the longest query's or
// the whole work over the resident warps or teams, whichever is more (a request
// loop's other batches add `load` queries of the batch's mean work). A team
// takes about 2.2 times fewer cycles per expansion than a warp (3,000 filtered
// int8 queries on 100k x 96 with 1-90 % selectivity: 2.1k against 4.6k), so it
// wins where the longest query decides (that batch: 55 against 143 ms) and
// loses where the SMs are full of queries of like length (592 teams or 2,368
// warps: 4,000 unfiltered queries at ef = 64 take 1.47 against 1.00 ms).
__global__ void __launch_bounds__(1024) query_order_kernel(SearchArgs a, uint32_t* order, uint8_t* bucket,
                                                           float warp_slots, float team_slots, float load,
                                                           uint32_t* route) {
    constexpr uint32_t B = 128;
    __shared__ uint32_t hist[B], next[B];
    __shared__ float wsum[32], wmax[32];
    for (uint32_t i = threadIdx.x; i < B; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    float sum = 0.0f, mx = 0.0f;
    for (uint32_t qi = threadIdx.x; qi < a.nq; qi += blockDim.x) {
        const float w = expected_work(a, qi);
        sum += w;
        mx = fmaxf(mx, w);
        const uint32_t bk = B - 1u - min(uint32_t(4.0f * log2f(w)), B - 1u);
        bucket[qi] = uint8_t(bk);
        atomicAdd(&hist[bk], 1u);
    }
    for (int off = 16; off > 0; off >>= 1) {
        sum += __shfl_xor_sync(kFull, sum, off);
        mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, off));
    }
    if ((threadIdx.x & 31) == 0) {
        wsum[threadIdx.x >> 5] = sum;
        wmax[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t at = 0;
        for (uint32_t i = 0; i < B; ++i) {
            next[i] = at;
            at += hist[i];
        }
        sum = mx = 0.0f;
        for (uint32_t i = 0; i < (blockDim.x >> 5); ++i) {
            sum += wsum[i];
            mx = fmaxf(mx, wmax[i]);
        }
        sum += sum * load / float(a.nq);
        *route = kTeamSpeed * fmaxf(mx, sum / warp_slots) > fmaxf(mx, sum / team_slots) ? kRouteTeam : kRouteWarp;
    }
    __syncthreads();
    for (uint32_t qi = threadIdx.x; qi < a.nq; qi += blockDim.x) order[atomicAdd(&next[bucket[qi]], 1u)] = qi;
}

}  // namespace dev

namespace {
using TeamKernel = void (*)(SearchArgs, TeamGeometry);
TeamKernel team_kernel(const SearchArgs& a) {
    if (a.quantized) return dev::search_team_kernel<dev::DK_ANY>;
    return a.ix.metric == 0 ? dev::search_team_kernel<dev::DK_L2> : dev::search_team_kernel<dev::DK_DOT>;
}
constexpr size_t kTeamSmemMax = 227 * 1024;
}  // namespace

cudaError_t plan_search_team(const SearchArgs& a, uint32_t ef_max, int num_sms, TeamGeometry* out) {
    TeamGeometry g;
    *out = g;
    if (a.ix.m0p > 64) return cudaSuccess;  // slots hold two masks
    g.ef_cap = std::min<uint32_t>(1024, std::max<uint32_t>(32, (ef_max + 31) / 32 * 32));
    // C: a power of two (its refills are sorted as one).
    g.cand_cap = 128;
    while (g.cand_cap < 2 * g.ef_cap) g.cand_cap <<= 1;
    // Eight warps; four when the batch is a little too large for two teams of
    // eight per SM and its queries are alike (592 queries on 200k x 128, ef =
    // 64: 410 us with four warps, 452 with eight, 622 with a warp per query;
    // one query: 238, 217 and 325 us; 16 warps were no faster).
    const bool alike = !a.efs && !a.filter_bits;
    g.warps = a.nq <= 2 * uint32_t(num_sms) || !alike ? 8 : 4;
    size_t off[8];
    const uint32_t words = ((a.ix.n + 31) / 32 + 3) & ~3u;
    const size_t base = dev::team_layout(a.ix.dp, a.ix.dc, a.ix.m0p, g, off);
    if (base > kTeamSmemMax) return cudaSuccess;
    // The visited bitmap in shared memory: up to 96 KB (two teams per SM), or
    // whatever fits when there is no more than one query per SM.
    const size_t room = a.nq <= uint32_t(num_sms) ? kTeamSmemMax - base : std::min(kTeamSmemMax - base, size_t(96) * 1024);
    if (size_t(words) * 4 + 16 <= room) g.bitmap_words = words;
    g.smem = dev::team_layout(a.ix.dp, a.ix.dc, a.ix.m0p, g, off);
    const TeamKernel kern = team_kernel(a);
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kern));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, int(32 * g.warps), g.smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaSuccess;
    g.resident = uint32_t(num_sms) * uint32_t(per_sm);
    g.blocks = std::min<uint32_t>(a.nq, g.resident);
    // Far lists: one entry per node at most, 256 MB in all (a query that
    // needs more goes to the retry pass).
    g.far_cap = std::min<uint32_t>((a.ix.n + 31) / 32 * 32, std::min<uint32_t>(1u << 18, (1u << 25) / g.blocks));
    *out = g;
    return cudaSuccess;
}

cudaError_t launch_search_team(const SearchArgs& a, const TeamGeometry& g, cudaStream_t stream) {
    team_kernel(a)<<<g.blocks, 32 * g.warps, g.smem, stream>>>(a, g);
    return cudaGetLastError();
}

cudaError_t launch_query_order(const SearchArgs& a, uint32_t* order, uint8_t* bucket, uint32_t warp_slots,
                               uint32_t team_slots, uint32_t load, uint32_t* route, cudaStream_t stream) {
    dev::query_order_kernel<<<1, 1024, 0, stream>>>(a, order, bucket, float(warp_slots), float(team_slots),
                                                    float(load), route);
    return cudaGetLastError();
}

}  // namespace hnswgpu
