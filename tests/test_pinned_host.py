"""The copies of pageable host arrays (sphg_pinned.h) on the CPU, against a small
stand-in for the CUDA runtime: a stream is a queue of operations that run only
when an event or a stream is waited for, so a copy that is not ordered after
the work before it moves the wrong bytes, every time."""
import os
import subprocess

import pytest

from sources_b200 import build

FAKE = r"""
#include "sphg_pinned.h"
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <functional>
#include <map>
#include <set>

// ------------------------------------------------------------ the stand-in
std::recursive_mutex M;
typedef std::pair<cudaStream_t, std::thread::id> Key;      // cudaStreamPerThread is another stream in each thread
std::map<Key, std::deque<std::function<void()>>> queues;
std::map<cudaEvent_t, std::pair<Key, size_t>> marks;       // event -> operations of its stream before it
std::map<Key, size_t> issued, done;
std::map<char*, size_t> pinned_mem;
std::set<std::thread::id> copiers;
std::set<const void*> device_ptrs;
char* dev_lo = nullptr; char* dev_hi = nullptr;
int fail_record = -1, freed_busy = 0;
size_t pending_pinned(const char* p) ;
Key key(cudaStream_t s) { return Key(s, s == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id()); }
void push(cudaStream_t s, std::function<void()> f) { queues[key(s)].push_back(f); ++issued[key(s)]; }
void run_to(Key k, size_t n) {
    while (done[k] < n) { queues[k].front()(); queues[k].pop_front(); ++done[k]; }
}
std::map<const char*, size_t> in_flight;                   // copies queued per page-locked buffer
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> l(M);
    *p = malloc(n); pinned_mem[(char*)*p] = n; return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::recursive_mutex> l(M);
    if (in_flight[(char*)p]) ++freed_busy;
    pinned_mem.erase((char*)p); free(p); return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::lock_guard<std::recursive_mutex> l(M); marks.erase(e); free((void*)e); return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::recursive_mutex> l(M);
    a->type = device_ptrs.count(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> l(M);
    copiers.insert(std::this_thread::get_id());
    const char* pin = (const char*)(kind == cudaMemcpyHostToDevice ? s : d);
    ++in_flight[pin];
    push(st, [=] { memcpy(d, s, n); --in_flight[pin]; });
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> l(M);
    if (fail_record >= 0 && fail_record-- == 0) return cudaErrorUnknown;
    marks[e] = {key(st), issued[key(st)]};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> l(M);
    if (marks.count(e)) run_to(marks[e].first, marks[e].second);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> l(M);
    run_to(key(s), issued[key(s)]);
    return cudaSuccess;
}
}

// -------------------------------------------------------------- the checks
int bad(const char* what) { printf("FAILED: %s\n", what); return 1; }
std::vector<PinnedCopies::Seg> segs(std::vector<std::vector<char>>& h) {
    std::vector<PinnedCopies::Seg> s;
    size_t off = 0;
    for (auto& v : h) { s.push_back({v.data(), nullptr, off, v.size()}); off += v.size(); }
    return s;
}
char val(size_t i) { return (char)(i * 7 + i / 251); }

// bytes through stream st: downwards after a kernel on st that writes the device range, upwards before one that reads it
int transfer(cudaStream_t st, size_t total, bool up, size_t* threads) {
    PinnedCopies pc;
    std::vector<std::vector<char>> h;
    for (size_t left = total; left;) { size_t n = std::min<size_t>(left, 1000003); h.emplace_back(n); left -= n; }
    std::vector<char> dev(total), got(total);
    copiers.clear();
    if (up) {
        size_t k = 0;
        for (auto& v : h) for (auto& c : v) c = val(k++);
    } else {
        std::lock_guard<std::recursive_mutex> l(M);
        push(st, [&] { for (size_t i = 0; i < total; ++i) dev[i] = val(i); });
    }
    if (pc.run(segs(h), dev.data(), total, up, st, 0) != 0) return bad("run");
    *threads = copiers.size();
    if (up) {
        { std::lock_guard<std::recursive_mutex> l(M); push(st, [&] { got = dev; }); }
        cudaStreamSynchronize(st);
    } else {
        size_t k = 0;
        for (auto& v : h) for (auto& c : v) got[k++] = c;
    }
    for (size_t i = 0; i < total; ++i) if (got[i] != val(i)) return bad("bytes");
    return 0;
}
"""

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture
def fake(tmp_path):
    """Compile the stand-in with a main() and run it."""
    def go(main):
        src, exe = tmp_path / "fake.cpp", tmp_path / "fake"
        src.write_text(FAKE + "int main() {\n" + main + "\nreturn 0;\n}\n")
        inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
        csrc = os.path.join(os.path.dirname(HERE), "sources_b200", "csrc")
        subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", inc, "-I", csrc, "-o", str(exe), str(src)], check=True)
        r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout == "", r.stdout + r.stderr
    return go


@pytest.mark.parametrize("up,total", [(0, 3 << 20), (0, 6 << 20), (1, 70 << 20)])
@pytest.mark.parametrize("stream", ["(cudaStream_t)64", "cudaStreamLegacy", "cudaStreamPerThread"])
def test_copies_follow_the_callers_stream(fake, stream, up, total):
    """Below and above the size from which helper threads share the work.  In another
    thread cudaStreamPerThread is another stream, so there the caller works alone, and
    leaves uploads to the driver."""
    mine = stream == "cudaStreamPerThread"
    if up and mine:
        fake(f"PinnedCopies pc; std::vector<std::vector<char>> h(1, std::vector<char>({total})); std::vector<char> d({total});"
             f"if (pc.run(segs(h), d.data(), {total}, true, {stream}, 0) != -1 || copiers.size()) return bad(\"taken\");")
        return
    alone = total < (4 << 20) or mine
    fake(f"size_t threads = 0; if (transfer({stream}, {total}, {up}, &threads)) return 1;"
         f"if (threads != {1 if alone else 4}) return bad(\"threads\");")


@pytest.mark.parametrize("up", [0, 1])
@pytest.mark.parametrize("record", [0, 1, 5, 17])
def test_a_failed_transfer_leaves_nothing_in_flight(fake, up, record):
    """The buffers go back to the pool when the call returns: no copy may still use one, whichever call failed."""
    fake(f"""const size_t total = 70 << 20;
    PinnedCopies pc;
    std::vector<std::vector<char>> h(1, std::vector<char>(total));
    std::vector<char> dev(total);
    fail_record = {record};
    if (pc.run(segs(h), dev.data(), total, {up}, (cudaStream_t)64, 0) != 1) return bad("status");
    for (auto& k : in_flight) if (k.second) return bad("a copy is in flight");
    size_t threads;
    if (transfer((cudaStream_t)65, total, {up}, &threads)) return 1;""")


def test_idle_buffers_serve_every_device(fake):
    """Eight pairs of buffers in all: those that one device's transfers made and left idle serve another's."""
    fake("""const size_t total = 6 << 20;
    PinnedCopies pc;
    for (int dev = 0; dev < 3; ++dev) {
        std::vector<PinnedCopies::Slot*> s;
        for (int i = 0; i < PinnedCopies::kSlots; ++i) {
            s.push_back(PinnedCopies::acquire(dev));
            if (!s.back() || s.back()->device != dev) return bad("no buffers");
        }
        if (PinnedCopies::acquire(dev) || PinnedCopies::acquire(dev + 1)) return bad("more buffers than the limit");
        if (pinned_mem.size() != 2 * PinnedCopies::kSlots) return bad("page-locked memory");
        for (auto* p : s) PinnedCopies::release(p);
    }
    std::vector<std::vector<char>> h(1, std::vector<char>(total));
    std::vector<char> dev(total);
    if (pc.run(segs(h), dev.data(), total, false, (cudaStream_t)64, 5) != 0) return bad("run");
    if (freed_busy) return bad("a buffer was freed with a copy in flight");""")


def test_idle_buffers_are_freed_after_their_copies(fake):
    """An upload returns with its last pieces queued; another device's transfer frees those buffers only then."""
    fake("""const size_t total = 70 << 20;
    PinnedCopies pc;
    std::vector<std::vector<char>> h(1, std::vector<char>(total));
    std::vector<char> dev(total);
    if (pc.run(segs(h), dev.data(), total, true, (cudaStream_t)64, 0) != 0) return bad("run");
    for (int i = 0; i < PinnedCopies::kSlots; ++i) if (!PinnedCopies::acquire(1)) return bad("no buffers");
    if (freed_busy) return bad("a buffer was freed with a copy in flight");""")


@pytest.mark.parametrize("up,total", [(0, 1 << 20), (1, 70 << 20)])
def test_device_arrays_stay_with_the_driver(fake, up, total):
    """A device address among the arrays is for the driver to move or refuse; the host never touches it."""
    fake(f"""PinnedCopies pc;
    std::vector<std::vector<char>> h(3, std::vector<char>({total}));
    std::vector<char> dev(3 * {total});
    auto s = segs(h);
    s[1].h0 = (char*)4096;
    device_ptrs.insert(s[1].h0);
    if (pc.run(s, dev.data(), dev.size(), {up}, (cudaStream_t)64, 0) != -1) return bad("taken");""")
