// Internals of the C ABI shared by capi.cpp and server.cpp: device buffers,
// per-call scratch slots, the index and brute-force handles, and the launch
// helper of one search.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "brute_tc.hpp"
#include "device.hpp"
#include "hnsw_gpu.h"
#include "host_index.hpp"

namespace hnswgpu {

// Records the message of the last failure on this thread; returns status.
int set_error(int status, const std::string& msg);
const char* last_error_text();
int from_err(const Err& e);
int cuda_fail(cudaError_t e, const char* where);

#define CU(call, where)                                      \
    do {                                                     \
        cudaError_t _e = (call);                             \
        if (_e != cudaSuccess) return ::hnswgpu::cuda_fail(_e, where); \
    } while (0)

inline uint32_t round_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

// Device allocations still to fail on purpose (hnsw_gpu_debug_fail_allocations):
// a host-side test hook for the out-of-device-memory paths.
inline std::atomic<int> g_fail_allocations{0};
// Visited-hash tags (hnsw_gpu_debug_visit_tags): 0 automatic, -1 off (32-bit
// ids), k > 0 an id space of at least k bits.
inline std::atomic<int> g_visit_tag_bits{0};
inline bool injected_alloc_failure() {
    int n = g_fail_allocations.load(std::memory_order_relaxed);
    while (n > 0)
        if (g_fail_allocations.compare_exchange_weak(n, n - 1, std::memory_order_relaxed)) return true;
    return false;
}

// Growable device buffer.
struct DBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t need) {
        if (need <= bytes) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        if (injected_alloc_failure()) return cudaErrorMemoryAllocation;  // as cudaMalloc: the old buffer is gone
        cudaError_t e = cudaMalloc(&p, need);
        if (e == cudaSuccess) bytes = need;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

// The outputs of one host-buffer call in one device buffer, so that they come
// back in one copy: keys and distances (nq rows of `stride`), counts,
// statuses, and `extra` more bytes of the caller's. Up to kStaged bytes go
// through pinned memory (a copy to pageable memory costs about 10 us however
// small it is: 1 query's four arrays took 40 of 183 us); larger ones, where
// the bytes decide, go to the caller's arrays directly. So does the first
// call's result: the driver pins 2 MB at a time, which costs 1.3 to 3 ms that only a
// handle that is used again gets back, unless another handle's buffer holds
// such a chunk already (a small buffer then takes about 5 us).
inline std::atomic<int> g_pinned_outputs{0};  // handles' pinned buffers alive
struct Outputs {
    static constexpr size_t kStaged = size_t(1) << 20, kSmall = size_t(1) << 18;
    DBuf dev;
    void* host = nullptr;
    size_t host_bytes = 0, rows = 0, stride = 0, tail = 0;
    bool cleared = false, used = false;
    uint64_t* keys() const { return dev.as<uint64_t>(); }
    float* dist() const { return reinterpret_cast<float*>(keys() + rows * stride); }
    uint32_t* count() const { return reinterpret_cast<uint32_t*>(dist() + rows * stride); }
    int32_t* status() const { return reinterpret_cast<int32_t*>(count() + rows); }
    uint32_t* extra() const { return reinterpret_cast<uint32_t*>(status() + rows); }
    size_t bytes() const { return rows * stride * 12 + rows * 8 + tail; }
    cudaError_t ensure(size_t nq, size_t row_stride, size_t extra_bytes = 0) {
        rows = nq;
        stride = row_stride;
        tail = extra_bytes;
        cleared = false;
        return dev.ensure(std::max<size_t>(bytes(), 16));
    }
    // The buffer holds what another call, of another shape, left there, so the
    // entries beyond a row's count are zeroed: on the device before a call
    // that will leave many (a k per query, a filter, k above the number of
    // rows; 1,000 queries for the best 1,000 of 300: 1.9 ms, 2.9 on the host),
    // else in the caller's arrays (failed queries; the scan of 10,000 counts
    // takes about 3 us).
    cudaError_t clear(cudaStream_t st) {
        cleared = true;
        return cudaMemsetAsync(dev.p, 0, rows * stride * 12, st);
    }
    void zero_unfilled(uint64_t* k, float* d, const uint32_t* c, const int32_t* s) const {
        for (size_t i = 0; i < rows; ++i) {
            const size_t n = s[i] == HNSW_OK ? c[i] : 0;
            if (n >= stride) continue;
            std::memset(k + i * stride + n, 0, (stride - n) * 8);
            std::memset(d + i * stride + n, 0, (stride - n) * 4);
        }
    }
    // Enqueues the copies, waits for the stream, and fills the caller's arrays
    // (`extra_out` with the extra bytes; `rows_out` false: no keys and distances).
    cudaError_t fetch(cudaStream_t st, uint64_t* k, float* d, uint32_t* c, int32_t* s, bool rows_out = true,
                      void* extra_out = nullptr) {
        const size_t kb = rows_out ? rows * stride * 8 : 0, db = rows_out ? rows * stride * 4 : 0;
        const bool staged =
            bytes() <= kStaged && (used || (bytes() <= kSmall && g_pinned_outputs.load(std::memory_order_relaxed) > 0));
        used = true;
        if (staged) {
            if (host_bytes < bytes()) {
                release_host();
                size_t want = 16384;
                while (want < bytes()) want <<= 1;
                if (cudaHostAlloc(&host, want, cudaHostAllocDefault) == cudaSuccess) {
                    host_bytes = want;
                    g_pinned_outputs.fetch_add(1, std::memory_order_relaxed);
                } else {
                    host = nullptr;
                    cudaGetLastError();  // no pinned memory: copy directly
                }
            }
            if (host_bytes >= bytes()) {
                cudaError_t e = cudaMemcpyAsync(host, dev.p, bytes(), cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                if (e != cudaSuccess) return e;
                const char* h = static_cast<const char*>(host);
                auto at = [&](const void* p) { return h + (static_cast<const char*>(p) - static_cast<const char*>(dev.p)); };
                if (kb) std::memcpy(k, at(keys()), kb);
                if (db) std::memcpy(d, at(dist()), db);
                std::memcpy(c, at(count()), rows * 4);
                std::memcpy(s, at(status()), rows * 4);
                if (extra_out) std::memcpy(extra_out, at(extra()), tail);
                if (rows_out && !cleared) zero_unfilled(k, d, c, s);
                return cudaSuccess;
            }
        }
        cudaError_t e = cudaSuccess;
        auto copy = [&](void* to, const void* from, size_t n) {
            if (e == cudaSuccess && n) e = cudaMemcpyAsync(to, from, n, cudaMemcpyDeviceToHost, st);
        };
        copy(c, count(), rows * 4);
        copy(s, status(), rows * 4);
        copy(k, keys(), kb);
        copy(d, dist(), db);
        if (extra_out) copy(extra_out, extra(), tail);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess && rows_out && !cleared) zero_unfilled(k, d, c, s);
        return e;
    }
    void release_host() {
        if (!host) return;
        cudaFreeHost(host);
        g_pinned_outputs.fetch_sub(1, std::memory_order_relaxed);
        host = nullptr;
        host_bytes = 0;
    }
    void release() {
        dev.release();
        release_host();
    }
};

// One concurrent call's stream and scratch.
struct Slot {
    cudaStream_t stream = nullptr;
    DBuf q, ks, efs, fbits, fused, fids, work, overflow, counters;
    hnswgpu::Outputs out;
    DBuf g_results, g_cands, g_visited;
    uint32_t g_warps = 0, g_ef_cap = 0, g_cand_cap = 0;
    uint64_t g_words = 0;
    DBuf spill_bits, spill_cands;  // persistent-mode spill areas (bitmaps kept zero)
    DBuf cold_pool, cold_tab; // cold candidate lists (persistent and retry warps)
    DBuf last_pool, last_tab, overflow2;  // last-resort pass (private cold regions)
    DBuf planned;                         // selectivity planner flags
    DBuf team_bits, team_far, order;      // team traversal: visited bitmaps, far candidates, query order
    size_t last_nq = 0;
    // Who took the last search: the warp kernel, teams, or whom the device's
    // route word (work[5]) names.
    enum { kWarps, kTeams, kDevice } taken_by = kWarps;
    ~Slot() {
        for (DBuf* b : {&q, &ks, &efs, &fbits, &fused, &fids, &work, &overflow, &counters,
                        &g_results, &g_cands, &g_visited, &spill_bits, &spill_cands, &cold_pool, &cold_tab, &last_pool,
                        &last_tab, &overflow2, &planned, &team_bits, &team_far, &order})
            b->release();
        out.release();
        if (stream) cudaStreamDestroy(stream);
    }
};

struct SlotPool {
    std::mutex mu;
    std::vector<std::unique_ptr<Slot>> free;
    int device = 0;
    int acquire(Slot** out) {
        {
            std::lock_guard<std::mutex> g(mu);
            if (!free.empty()) {
                *out = free.back().release();
                free.pop_back();
                return HNSW_OK;
            }
        }
        auto* s = new (std::nothrow) Slot();
        if (!s) return set_error(HNSW_ERR_INVALID_ARGUMENT, "out of host memory");
        cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            delete s;
            return cuda_fail(e, "cudaStreamCreate");
        }
        *out = s;
        return HNSW_OK;
    }
    void release(Slot* s) {
        std::lock_guard<std::mutex> g(mu);
        free.emplace_back(s);
    }
};

// A named range on the NVTX timeline around a host-side phase (staging,
// enqueue, copies, a build wave). Profilers that attach an NVTX tool (Nsight
// Systems, Nsight Compute with --nvtx) show it; without one it costs a
// function call.
struct TraceRange {
    explicit TraceRange(const char* name) { nvtxRangePushA(name); }
    ~TraceRange() { nvtxRangePop(); }
    TraceRange(const TraceRange&) = delete;
    TraceRange& operator=(const TraceRange&) = delete;
};

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

// Scratch geometry per (ef bound): results, candidates and the visited
// hash sized so that a typical traversal at that ef stays in shared memory.
// Queries whose ef exceeds the fast kernel's 1024 go to the retry pass.
SearchGeometry pick_geometry(uint32_t ef_max, uint32_t dp, uint32_t dc, bool persistent, bool filtered, uint32_t n);

}  // namespace hnswgpu

// The handle types of the C ABI (opaque to callers).
using hnswgpu::DBuf;
using hnswgpu::DeviceGuard;
using hnswgpu::DeviceIndexView;
using hnswgpu::Slot;
using hnswgpu::SlotPool;
using hnswgpu::Builder;

struct hnsw_gpu_index {
    int device = 0;
    int num_sms = 148;
    hnsw_index_info info{};
    DeviceIndexView view;
    DBuf vec, codes, norms, offset, adj0, upoff, adjU, keys, dead;
    SlotPool slots;
    bool counters = false;
    std::mutex counters_mu;
    std::vector<uint32_t> last_counters;
    // Scratch of the device-pointer entry point: one slot, ordered on the
    // device (an event joins each call after the previous one).
    std::mutex dev_mu;
    std::unique_ptr<Slot> dev_slot;
    // Fixed schedule (hnsw_gpu_set_schedule); ef_cap == 0 means automatic.
    hnswgpu::SearchGeometry fixed{0, 0, 0, 0, 0};
    // Autotuned schedules (hnsw_gpu_autotune) per ef bucket, bucket b
    // covering max(ef, k) in (32(b-1), 32b], b = 1..32 (the last one also
    // everything above 1024), one per mode; ef_cap == 0 means not tuned.
    // `mode` is the faster mode of the bucket (-1: not tuned).
    struct Tuned {
        hnswgpu::SearchGeometry geo[2] = {{0, 0, 0, 0, 0}, {0, 0, 0, 0, 0}};
        int32_t mode = -1;
    };
    std::mutex tune_mu;
    Tuned tuned[33];
    // The occupancy heuristic's choices (pick_geometry, about twenty occupancy
    // queries) by ef capacity, mode, filter and visited-tag setting.
    std::mutex plan_mu;
    std::map<uint64_t, hnswgpu::SearchGeometry> plans;
    cudaEvent_t dev_done = nullptr;
    // Tensor-core traversal rows, built on first use (tc_mu): BF16 high
    // parts, low parts (BF16X3), f32 squared norms (L2).
    std::mutex tc_mu;
    DBuf tc_hi, tc_lo, tc_norm;
    DBuf chk;  // bounds-check word of the checked build (2 x u32)
    bool tc_hi_ready = false, tc_lo_ready = false;
    ~hnsw_gpu_index() {
        DeviceGuard g(device);
        if (dev_done) {
            cudaEventSynchronize(dev_done);
            cudaEventDestroy(dev_done);
        }
        dev_slot.reset();
        for (DBuf* b : {&vec, &codes, &norms, &offset, &adj0, &upoff, &adjU, &keys, &dead, &tc_hi, &tc_lo, &tc_norm, &chk})
            b->release();
        std::lock_guard<std::mutex> l(slots.mu);
        slots.free.clear();
    }
};

struct hnsw_gpu_brute {
    int device = 0;
    int num_sms = 148;
    uint32_t n = 0, dim = 0, dp = 0;
    int metric = 0;
    float max_xnorm = 0.0f;  // largest row norm (error margins of the tensor-core path)
    DBuf base, keys;
    DBuf krank, skeys;  // key ranks and sorted keys, when the keys do not ascend
    SlotPool slots;
    std::mutex mu;
    DBuf qprep, part, minima, q;
    hnswgpu::Outputs out;
    DBuf fbits, fused, fids, rows;  // filter bitmaps, flags, bitmap ids and admitted rows of a filtered search
    // Tensor-core path: BF16 operand rows per term count (index 0: 1 term, 1: 3 terms).
    DBuf bop[2], xnorm2;
    uint32_t bop_kp[2] = {0, 0};
    DBuf aop, dense, thr1, thr2, margin, qnorm2, cand;
    uint64_t last_candidates = 0, last_queries = 0;
    float last_ms[4] = {0, 0, 0, 0};
    long long wait_budget = 4000000000ll;  // tensor-core pipeline waits, clock cycles
    uint32_t stall = 0;                    // test switch: the MMA issuer's wait runs out
    uint32_t tc_pairs = 0;                 // paired (cta_group::2) tensor-core kernel
    cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    cudaStream_t stream = nullptr;
    ~hnsw_gpu_brute() {
        DeviceGuard g(device);
        for (DBuf* b : {&base, &keys, &krank, &skeys, &qprep, &part, &minima, &q, &fbits, &fused, &fids, &rows,
                        &bop[0], &bop[1], &xnorm2,
                        &aop, &dense, &thr1, &thr2, &margin, &qnorm2, &cand})
            b->release();
        out.release();
        for (cudaEvent_t& e : ev)
            if (e) cudaEventDestroy(e);
        if (stream) cudaStreamDestroy(stream);
    }
};

struct hnsw_builder {
    std::unique_ptr<Builder> b;
    hnsw_gpu_build_stats last{};  // figures of the last device link
};

namespace hnswgpu {
// Enqueues one search on `stream` with device pointers. ef_max bounds every
// per-query max(ef, k) of the batch; `load` is the number of queries of other
// batches that run beside it. With `reserve` it only grows the slot's buffers to
// what that search needs.
int enqueue_search(hnsw_gpu_index* gi, Slot* s, const float* d_q, size_t nq, const hnsw_search_opts& o,
                   const uint32_t* d_ks, const uint32_t* d_efs, const uint64_t* d_fbits, const uint8_t* d_fused,
                   const uint32_t* d_fids, uint64_t* d_keys, float* d_dist, uint32_t* d_count, int32_t* d_status, uint32_t ef_max,
                   uint32_t out_stride, cudaStream_t stream, const SearchGeometry* force = nullptr,
                   bool publish = false, uint32_t load = 0, bool reserve = false);
int reserve_search(hnsw_gpu_index* gi, Slot* s, uint32_t max_nq, uint32_t max_ef, const hnsw_search_opts& o,
                   bool filtered);
// The ef bucket of the tuning table for a batch whose max(ef, k) is ef_max.
inline uint32_t tune_bucket(uint32_t ef_max) {
    return ef_max > 1024 ? 32u : std::max<uint32_t>(1, (ef_max + 31) / 32);
}
}  // namespace hnswgpu
