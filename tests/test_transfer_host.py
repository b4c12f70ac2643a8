"""The pinned-slot transfers (csrc/transfer.cu) on the CPU, compiled against a
stand-in for the CUDA runtime whose copies run as late as their stream allows:
a slot refilled, emptied or given back too early shows as wrong bytes or as a
copy left behind.  Allocations, thread starts and event records that fail must
neither end the process nor lose bytes."""
import subprocess

import pytest

from conftest import ROOT

RUNTIME = r"""
#pragma once
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
enum { cudaEventDisableTiming = 2, cudaHostAllocPortable = 1, cudaMemoryTypeUnregistered = 0 };
struct cudaPointerAttributes { int type; };
struct Copy { void* d; const void* h; size_t n; };
struct Stream {
    std::mutex mu;
    std::vector<Copy> work;  // reserved: the runtime stand-in allocates nothing here
    size_t ran = 0, records_left = ~size_t(0);  // event records before one fails
    void run(size_t n) { for (; ran < n; ran++) std::memcpy(work[ran].d, work[ran].h, work[ran].n); }
};
struct Event { Stream* s = nullptr; size_t after = 0; };
typedef Stream* cudaStream_t;
typedef Event* cudaEvent_t;
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = 0; return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, int) { *p = std::malloc(n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = static_cast<Event*>(std::calloc(1, sizeof(Event))); return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* h, size_t n, cudaMemcpyKind, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(s->mu);
    s->work.push_back({d, h, n});
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(s->mu);
    if (s->records_left-- == 0) return cudaErrorUnknown;
    e->s = s;
    e->after = s->work.size();
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (!e->s) return cudaSuccess;  // never recorded
    std::lock_guard<std::mutex> lk(e->s->mu);
    e->s->run(e->after);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::mutex> lk(s->mu);
    s->run(s->work.size());
    return cudaSuccess;
}
"""

HARNESS = r"""
#include <cstdio>
#include <new>
#include <string>
#include <thread>
#include "transfer.h"
thread_local int news_left = -1;  // allocations of this thread before every further one fails
void* operator new(size_t n) {
    if (news_left == 0) throw std::bad_alloc();
    if (news_left > 0) news_left--;
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
unsigned std::thread::hardware_concurrency() noexcept { return 16; }
static std::vector<char> host, dev, back;
static void fill(int seed) {
    for (size_t i = 0; i < host.size(); i++) host[i] = char(i * 31 + i / 4096 + seed);
    dev.assign(host.size(), 0);
    back.assign(host.size(), 0);
}
static int check(bool ok, const char* what) {
    if (!ok) std::printf("%s\n", what);
    return ok ? 0 : 1;
}
int main(int, char** argv) {
    const std::string mode = argv[1];
    if (mode == "no memory for a user") news_left = 0;
    ym::transfer_retain();
    news_left = -1;
    Stream st;
    st.work.reserve(4096);
    host.resize((size_t(37) << 20) / 2 + 12345);  // a partial last chunk
    int bad = 0;
    for (int k = 0; k < 12; k++) {  // the first ones go to the driver, then the slots are there
        fill(k);
        if (mode == "no memory for threads" && k >= 10) news_left = k - 10;
        cudaError_t e = ym::transfer_upload(0, dev.data(), host.data(), host.size(), &st);
        const bool via_slots = st.ran > 0 && st.ran == st.work.size();
        bad += check(e == cudaSuccess, "upload status");
        cudaStreamSynchronize(&st);
        bad += check(dev == host, "upload bytes");
        e = ym::transfer_download(0, back.data(), dev.data(), host.size(), &st);
        news_left = -1;
        bad += check(e == cudaSuccess, "download status");
        cudaStreamSynchronize(&st);
        bad += check(back == host, "download bytes");
        if (k == 11) bad += check(via_slots, "the slots were not used");
        st.work.clear();
        st.ran = 0;
    }
    if (mode == "no event record")
        for (size_t n = 0; n < 40; n += 3)
            for (int down = 0; down < 2; down++) {
                st.records_left = n;
                const cudaError_t e = down ? ym::transfer_download(0, back.data(), dev.data(), host.size(), &st)
                                           : ym::transfer_upload(0, dev.data(), host.data(), host.size(), &st);
                st.records_left = ~size_t(0);
                bad += check((e == cudaSuccess) == (n >= 19), "status");  // 19 chunks
                bad += check(st.ran == st.work.size(), "a copy is left in the slots");
                st.work.clear();
                st.ran = 0;
            }
    ym::transfer_release();
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("transfer")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "main.cpp").write_text(HARNESS)
    csrc = ROOT / "latticeyangmills_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(d), "-I", str(csrc), "-x", "c++",
                    str(csrc / "transfer.cu"), str(d / "main.cpp"), "-o", str(d / "harness")], check=True)
    return d / "harness"


@pytest.mark.parametrize("mode", ["plain", "no memory for a user", "no memory for threads", "no event record"])
def test_transfers_are_exact_and_do_not_throw(harness, mode):
    res = subprocess.run([str(harness), mode], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, (res.returncode, res.stdout, res.stderr)
