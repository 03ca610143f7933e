// Copies between the caller's pageable host arrays and the device.
//
// cudaMemcpyAsync moves pageable memory through the driver's own pinned buffer on the calling thread;
// for a solve's result it also takes the page faults of an array that nobody has touched yet, one at a
// time. Large copies go through a pinned buffer of this library instead, up to kThreads host threads
// (fewer where the caller's OpenMP setting says so) each with two slots of kPiece bytes: one slot is
// copied by the host while the other is on the link. The host's share is bound by its memory
// bandwidth, so four threads, not all cores.
//
// 21.5 MB (42,048 nodes x 64 columns), potentials at 1,000 probes, whole call: 2.1 -> 1.2 ms; the refined
// solve's 21.5 MB into a fresh array: 38.9 -> 37.8 ms.
#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <vector>

#include "solver.h"

namespace bie {
namespace {

constexpr int kThreads = 4, kSlots = 2 * kThreads;
constexpr size_t kPiece = size_t(512) << 10;
constexpr size_t kStaged = size_t(2) << 20;  // smaller copies are the driver's: a thread team costs about 10 us
constexpr size_t kKept = 4;                  // pinned buffers (4 MB each) kept between calls

struct Stage {
    int device = -1;
    char* buf = nullptr;         // kSlots pieces, pinned
    cudaEvent_t ev[kSlots] = {};  // the last copy out of or into a slot
};

std::mutex g_mu;
std::vector<Stage*> g_free;

void destroy(Stage* st) {
    for (cudaEvent_t e : st->ev)
        if (e) {
            cudaEventSynchronize(e);
            cudaEventDestroy(e);
        }
    if (st->buf) cudaFreeHost(st->buf);
    delete st;
}

// A stage of the current device, or null when none can be had (no pinned memory left).
Stage* acquire(int device) {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        for (size_t i = 0; i < g_free.size(); ++i)
            if (g_free[i]->device == device) {
                Stage* st = g_free[i];
                g_free.erase(g_free.begin() + i);
                return st;
            }
    }
    Stage* st = new Stage;
    st->device = device;
    bool ok = cudaMallocHost((void**)&st->buf, kSlots * kPiece) == cudaSuccess;
    for (cudaEvent_t& e : st->ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (ok) return st;
    cudaGetLastError();
    destroy(st);
    return nullptr;
}

void give_back(Stage* st) {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_free.size() < kKept) {
            g_free.push_back(st);
            return;
        }
    }
    destroy(st);
}

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Copies `bytes` between dev and host through the stage, pieces dealt out to the threads in turn. A slot
// is written again only once its event says that the link has read it (or the host has, on the way out).
cudaError_t staged(bool in, char* dev, char* host, size_t bytes, Stage* st, cudaStream_t s) {
    const int64_t pieces = (int64_t)((bytes + kPiece - 1) / kPiece);
    std::atomic<int> err{(int)cudaSuccess};
#pragma omp parallel num_threads(std::min(kThreads, omp_get_max_threads()))
    {
        const int t = omp_get_thread_num(), nt = omp_get_num_threads();
        auto ck = [&](cudaError_t e) {
            if (e != cudaSuccess) err.store((int)e);
            return e == cudaSuccess && err.load() == (int)cudaSuccess;
        };
        int prev = -1;
        cudaGetDevice(&prev);
        bool ok = ck(cudaSetDevice(st->device));
        auto len = [&](int64_t p) { return std::min(kPiece, bytes - (size_t)p * kPiece); };
        auto slot = [&](int64_t u) { return 2 * t + (int)(u & 1); };
        const int64_t mine = t < pieces ? (pieces - t + nt - 1) / nt : 0;  // pieces t, t + nt, ...
        if (in) {
            for (int64_t u = 0; u < mine && ok; ++u) {
                const int64_t p = t + u * nt;
                char* b = st->buf + (size_t)slot(u) * kPiece;
                if (!(ok = ck(cudaEventSynchronize(st->ev[slot(u)])))) break;
                std::memcpy(b, host + (size_t)p * kPiece, len(p));
                ok = ck(cudaMemcpyAsync(dev + (size_t)p * kPiece, b, len(p), cudaMemcpyHostToDevice, s)) &&
                     ck(cudaEventRecord(st->ev[slot(u)], s));
            }
        } else {
            auto fetch = [&](int64_t u) {
                const int64_t p = t + u * nt;
                return ck(cudaEventSynchronize(st->ev[slot(u)])) &&
                       ck(cudaMemcpyAsync(st->buf + (size_t)slot(u) * kPiece, dev + (size_t)p * kPiece, len(p),
                                          cudaMemcpyDeviceToHost, s)) &&
                       ck(cudaEventRecord(st->ev[slot(u)], s));
            };
            for (int64_t u = 0; u < std::min<int64_t>(2, mine) && ok; ++u) ok = fetch(u);
            for (int64_t u = 0; u < mine && ok; ++u) {
                const int64_t p = t + u * nt;
                if (!(ok = ck(cudaEventSynchronize(st->ev[slot(u)])))) break;
                std::memcpy(host + (size_t)p * kPiece, st->buf + (size_t)slot(u) * kPiece, len(p));
                if (u + 2 < mine) ok = fetch(u + 2);
            }
        }
        if (prev >= 0 && prev != st->device) cudaSetDevice(prev);
    }
    return (cudaError_t)err.load();
}

void copy(bool in, void* dev, void* host, size_t bytes, cudaStream_t s) {
    int device = 0;
    BIE_CK(cudaGetDevice(&device));
    Stage* st = bytes >= kStaged && pageable(host) ? acquire(device) : nullptr;
    if (!st) {
        BIE_CK(cudaMemcpyAsync(in ? dev : host, in ? host : dev, bytes, in ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, s));
        return;
    }
    const cudaError_t e = staged(in, (char*)dev, (char*)host, bytes, st, s);
    if (e != cudaSuccess) {
        destroy(st);
        BIE_CK(e);
    }
    give_back(st);
}

}  // namespace

void copy_in(void* dev, const void* host, size_t bytes, cudaStream_t s) { copy(true, dev, const_cast<void*>(host), bytes, s); }
void copy_out(void* host, const void* dev, size_t bytes, cudaStream_t s) { copy(false, const_cast<void*>(dev), host, bytes, s); }

void copy_release() {
    std::vector<Stage*> all;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        while (g_free.size() > 1) {
            all.push_back(g_free.back());
            g_free.pop_back();
        }
    }
    for (Stage* st : all) destroy(st);
}

}  // namespace bie
