// hj_hostcopy.cu - host relations to the device.
//
// A copy from pageable memory goes through the driver's own staging on one thread, at about 10 GB/s of the
// ~55 GB/s the link carries: 8.1 ms of an 8.2 ms join of 2^20 x 2^22 host tuples. Here up to kCopyThreads
// threads of the call copy 2 MB pieces into page-locked buffers, two per thread, and issue the pieces'
// copies on the join's stream: 2.4 to 2.8 ms for the same join, whole calls on different machines (on the one where
// it took 2.4: 3 threads 2.9, 6 threads 2.5, 12 threads of 1 MB pieces 3.9, which then wait for each other in the
// driver). The buffers (16 MB) belong to the context, are allocated by its first large pageable copy and freed
// with it; the threads end before the call goes on. Page-locked sources, and copies too small to repay the
// threads, take the plain copy, and so does a call that cannot get buffers; fewer threads copy more pieces each.
#include <atomic>
#include <cstring>
#include <thread>

#include "hj_ctx.h"
#include "hj_internal.h"

namespace hj {

namespace {

constexpr int kCopyThreads = 4, kCopyBuffers = 2 * kCopyThreads;
static_assert(kCopyBuffers == hj_ctx::kCopyEvents, "an event per buffer");
constexpr size_t kCopyPiece = 2u << 20, kCopyMin = 4u << 20;
constexpr int kMaxCopies = 2;

bool pageable(const void *p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

bool get_buffers(hj_ctx *c) {
    if (c->copy_buf) return true;
    if (cudaMallocHost(&c->copy_buf, kCopyBuffers * kCopyPiece) != cudaSuccess) {
        cudaGetLastError();
        c->copy_buf = nullptr;
        return false;
    }
    for (cudaEvent_t &ev : c->copy_ev) {
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            ev = nullptr;
            free_copy_buffers(c);
            return false;
        }
    }
    return true;
}

}  // namespace

void free_copy_buffers(hj_ctx *c) {
    for (cudaEvent_t &ev : c->copy_ev) {
        if (ev) cudaEventDestroy(ev);
        ev = nullptr;
    }
    if (c->copy_buf) cudaFreeHost(c->copy_buf);
    c->copy_buf = nullptr;
}

int copy_in(hj_ctx *c, const HostCopy *copies, int ncopies, bool pinned, cudaStream_t st) {
    size_t first[kMaxCopies + 1] = {};  // pieces of the copies before
    size_t staged = 0;
    bool slow[kMaxCopies] = {};
    if (ncopies > kMaxCopies) return HJ_E_INVAL;
    for (int k = 0; k < ncopies; k++) {
        slow[k] = !pinned && pageable(copies[k].src);
        if (slow[k]) staged += copies[k].bytes;
    }
    const bool stage = staged >= kCopyMin && get_buffers(c);
    for (int k = 0; k < ncopies; k++) {
        slow[k] = slow[k] && stage;
        first[k + 1] = first[k] + (slow[k] ? (copies[k].bytes + kCopyPiece - 1) / kCopyPiece : 0);
        if (!slow[k] &&
            cudaMemcpyAsync(copies[k].dst, copies[k].src, copies[k].bytes, cudaMemcpyHostToDevice, st) != cudaSuccess)
            return HJ_E_DEVICE;
    }
    const size_t pieces = first[ncopies];
    if (!pieces) return HJ_OK;
    std::atomic<size_t> next{0};
    std::atomic<int> bad{0};
    auto work = [&](int w) {
        if (cudaSetDevice(c->device) != cudaSuccess) {
            bad = 1;
            return;
        }
        for (int turn = 0;; turn ^= 1) {
            const size_t i = next.fetch_add(1);
            if (i >= pieces || bad) return;
            const int b = 2 * w + turn;
            char *buf = c->copy_buf + (size_t)b * kCopyPiece;
            int k = 0;
            while (i >= first[k + 1]) k++;
            const HostCopy &cp = copies[k];
            const size_t off = (i - first[k]) * kCopyPiece, n = cp.bytes - off < kCopyPiece ? cp.bytes - off : kCopyPiece;
            // The copy that last read this buffer (of this call or an earlier one) has to be done.
            if (cudaEventSynchronize(c->copy_ev[b]) != cudaSuccess) {
                bad = 1;
                return;
            }
            memcpy(buf, static_cast<const char *>(cp.src) + off, n);
            if (cudaMemcpyAsync(static_cast<char *>(cp.dst) + off, buf, n, cudaMemcpyHostToDevice, st) != cudaSuccess ||
                cudaEventRecord(c->copy_ev[b], st) != cudaSuccess) {
                bad = 1;
                return;
            }
        }
    };
    const unsigned cores = std::thread::hardware_concurrency();
    const int want = cores < 2 ? 1 : cores < (unsigned)kCopyThreads ? (int)cores : kCopyThreads;
    std::thread threads[kCopyThreads];
    int started = 1;
    try {
        for (; started < want; started++) threads[started] = std::thread(work, started);
    } catch (...) {  // no more threads (or memory for them): those that started, and this one, do all pieces
    }
    work(0);
    for (int w = 1; w < started; w++) threads[w].join();
    return bad ? HJ_E_DEVICE : HJ_OK;
}

}  // namespace hj
