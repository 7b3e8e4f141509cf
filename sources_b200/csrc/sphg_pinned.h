// sphg_pinned.h — host <-> device copies of pageable host arrays (host code only).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace {

// Host <-> device copies of pageable host arrays through a small page-locked
// buffer of the library's own.  A pageable cudaMemcpyAsync stages through the
// driver one array at a time and, downwards, waits for each (18 us an array
// however small); here the arrays of a transfer are cut into pieces of one
// contiguous device range, copied by the host into or out of the buffer, and
// moved by one DMA per piece.  From kThreadBytes up, kWorkers host threads (made
// for the transfer and joined before it returns) take turns, which also
// spreads the page faults of arrays never touched before.
// Measured on a 16-core host, through the driver -> through this buffer:
// download of 4,008 particles 564 -> 168 us, 58,858 particles 2.26 -> 1.27 ms
// (3.8 -> 2.8 ms into new arrays), 912,016 particles 17.6 -> 10.5 ms (90 -> 35
// ms into new arrays); upload of 912,016 particles 16.5 -> 11.8 ms.  Below
// kUpBytes uploads stay with the driver, whose copies of arrays in use are
// as fast or faster (58,858 particles: 1.16 ms against 1.69).  Pieces of 2 MB
// move the largest transfers 20 % faster but cost a new context 5 ms more.
struct PinnedCopies {
    struct Seg { char* h0; char* h1; size_t off, bytes; };   // host array (and a second one, downwards), its device range
    static constexpr size_t kPiece = 512 << 10, kThreadBytes = 4 << 20, kUpBytes = 64 << 20;
    static constexpr int kWorkers = 4;
    // One worker's two buffers, lent to one transfer at a time.  The slots are
    // shared by the contexts of the process (making one takes as long as ten
    // small transfers), at most kSlots of them, and freed with the last context.
    // At the limit an idle slot of another device gives way to a new one.
    struct Slot {
        int device = 0;
        char* buf[2] = {nullptr, nullptr};
        cudaEvent_t ev[2] = {nullptr, nullptr};
    };
    static constexpr int kSlots = 2 * kWorkers;
    struct Pool {
        std::mutex m;
        std::vector<Slot*> idle;
        int made = 0, users = 0;
    };
    static Pool& pool() {
        static Pool* p = new Pool();   // never destroyed: a context may outlive the statics
        return *p;
    }
    static void destroy(Slot* s) {
        for (int b = 0; b < 2; ++b) {
            if (s->ev[b]) {
                cudaEventSynchronize(s->ev[b]);   // the last pieces of an upload may still be queued
                cudaEventDestroy(s->ev[b]);
            }
            if (s->buf[b]) cudaFreeHost(s->buf[b]);
        }
        delete s;
    }
    static Slot* acquire(int device) {
        Pool& P = pool();
        Slot* other = nullptr;
        {
            std::lock_guard<std::mutex> l(P.m);
            for (size_t i = 0; i < P.idle.size(); ++i)
                if (P.idle[i]->device == device) {
                    Slot* s = P.idle[i];
                    P.idle.erase(P.idle.begin() + (long)i);
                    return s;
                }
            if (P.made < kSlots) {
                ++P.made;
            } else {
                if (P.idle.empty()) return nullptr;
                other = P.idle.back();
                P.idle.pop_back();
            }
        }
        if (other) destroy(other);
        Slot* s = new Slot();
        s->device = device;
        bool ok = true;
        for (int b = 0; b < 2 && ok; ++b) {
            void* q = nullptr;
            ok = cudaHostAlloc(&q, kPiece, cudaHostAllocDefault) == cudaSuccess;
            s->buf[b] = (char*)q;
            ok = ok && cudaEventCreateWithFlags(&s->ev[b], cudaEventDisableTiming) == cudaSuccess;
        }
        if (ok) return s;
        cudaGetLastError();
        destroy(s);
        std::lock_guard<std::mutex> l(P.m);
        --P.made;
        return nullptr;
    }
    static void release(Slot* s) {
        Pool& P = pool();
        std::lock_guard<std::mutex> l(P.m);
        P.idle.push_back(s);
    }
    PinnedCopies() {
        std::lock_guard<std::mutex> l(pool().m);
        ++pool().users;
    }
    ~PinnedCopies() {
        Pool& P = pool();
        std::lock_guard<std::mutex> l(P.m);
        if (--P.users > 0) return;
        for (Slot* s : P.idle) destroy(s);
        P.made -= (int)P.idle.size();
        P.idle.clear();
    }
    PinnedCopies(const PinnedCopies&) = delete;
    PinnedCopies& operator=(const PinnedCopies&) = delete;
    static cudaMemoryType type(const void* p) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return cudaMemoryTypeUnregistered; }
        return a.type;
    }
    // host side of bytes [o, o + n) of the device range
    static void host_part(const std::vector<Seg>& s, size_t o, size_t n, char* pin, bool up) {
        for (const Seg& g : s) {
            if (g.off + g.bytes <= o || g.off >= o + n) continue;
            const size_t b = std::max(o, g.off), e = std::min(o + n, g.off + g.bytes);
            if (up) {
                memcpy(pin + (b - o), g.h0 + (b - g.off), e - b);
            } else {
                if (g.h0) memcpy(g.h0 + (b - g.off), pin + (b - o), e - b);
                if (g.h1) memcpy(g.h1 + (b - g.off), pin + (b - o), e - b);
            }
        }
    }
    // pieces w, w + nw, .. of the transfer
    static int work(Slot* slot, int w, int nw, const std::vector<Seg>& s, char* dev, size_t total, size_t piece, bool up,
                    cudaStream_t st) {
        if (cudaSetDevice(slot->device) != cudaSuccess) return 1;
        char** buf = slot->buf;
        cudaEvent_t* ev = slot->ev;
        const size_t np = (total + piece - 1) / piece;
        int used = 0;
        size_t prev = 0;
        bool pending = false;
        for (size_t i = (size_t)w; i < np; i += (size_t)nw, ++used) {
            const int b = used & 1;
            const size_t o = i * piece, n = std::min(piece, total - o);
            // the buffer's last piece (of this transfer or an earlier one) has left
            if (cudaEventSynchronize(ev[b]) != cudaSuccess) return 1;
            if (up) {
                host_part(s, o, n, buf[b], true);
                if (cudaMemcpyAsync(dev + o, buf[b], n, cudaMemcpyHostToDevice, st) != cudaSuccess) return 1;
                if (cudaEventRecord(ev[b], st) != cudaSuccess) return 1;
            } else {
                if (cudaMemcpyAsync(buf[b], dev + o, n, cudaMemcpyDeviceToHost, st) != cudaSuccess) return 1;
                if (cudaEventRecord(ev[b], st) != cudaSuccess) return 1;
                if (pending && drain(slot, b ^ 1, s, prev, std::min(piece, total - prev))) return 1;
                prev = o;
                pending = true;
            }
        }
        return pending ? drain(slot, (used - 1) & 1, s, prev, std::min(piece, total - prev)) : 0;
    }
    static int drain(Slot* slot, int b, const std::vector<Seg>& s, size_t o, size_t n) {
        if (cudaEventSynchronize(slot->ev[b]) != cudaSuccess) return 1;
        host_part(s, o, n, slot->buf[b], false);
        return 0;
    }
    // 0 done (upwards: the host arrays are no longer read), 1 error, -1 not taken (page-locked arrays only, a
    // device address among them, or no buffer)
    int run(const std::vector<Seg>& s, char* dev, size_t total, bool up, cudaStream_t st, int device) {
        // cudaStreamPerThread is another stream in each thread: the calling thread then works alone, and uploads,
        // which one thread moves no faster than the driver, stay with the driver
        const bool shared = st != cudaStreamPerThread;
        if (total == 0 || (up && (total < kUpBytes || !shared))) return -1;
        bool any = false;
        for (const Seg& g : s) {
            for (const char* h : {g.h0, g.h1}) {
                const cudaMemoryType t = h ? type(h) : cudaMemoryTypeHost;
                if (t == cudaMemoryTypeDevice) return -1;
                any = any || t == cudaMemoryTypeUnregistered;
            }
        }
        if (!any) return -1;
        Slot* slot[kWorkers];
        int nw = 0;
        for (const int want = total >= kThreadBytes && shared ? kWorkers : 1; nw < want; ++nw)
            if (!(slot[nw] = acquire(device))) break;
        if (nw == 0) return -1;
        const size_t piece = std::min(kPiece, (total + 255) / 256 * 256);
        std::atomic<int> bad{0};
        std::thread th[kWorkers];
        int here = 1;   // worker 0 is this thread, and stands in for threads that could not be made
        for (int w = 1; w < nw; ++w) {
            try {
                th[w] = std::thread([&, w] { if (work(slot[w], w, nw, s, dev, total, piece, up, st)) bad = 1; });
            } catch (...) {
                here |= 1 << w;
            }
        }
        for (int w = 0; w < nw; ++w)
            if ((here >> w & 1) && work(slot[w], w, nw, s, dev, total, piece, up, st)) bad = 1;
        for (int w = 1; w < nw; ++w)
            if (th[w].joinable()) th[w].join();
        if (bad) cudaStreamSynchronize(st);   // a copy may be in flight whose event was not recorded
        for (int w = 0; w < nw; ++w) release(slot[w]);
        return bad;
    }
};

}  // namespace
