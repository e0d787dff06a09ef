// A CUDA runtime without a device, for the library's host code (csrc/api.cu, host_copy.cu, commit_api.cu): device memory is heap memory, and a
// stream's work is done only when something waits for it, so that whatever relies on a copy being "probably through" shows.
//   fail_at   the how-manyth fallible call from now on fails (-1: none)
//   faults    what went wrong: memory freed under a copy of another stream, a copy to or from memory that is gone
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <deque>
#include <map>
#include <string>
#include <vector>

namespace fake {

struct Event;
struct Op { char* to; const char* from; size_t bytes; std::vector<char> held; Event* wait; unsigned long long upto; };
struct Stream { std::deque<Op> q; unsigned long long issued = 0, done = 0; };
struct Event { Stream* s = nullptr; unsigned long long seq = 0; };

inline std::vector<Stream*> streams;
inline std::map<const char*, size_t> device, locked;  // start -> bytes
inline std::vector<std::string> faults;
inline long fail_at = -1, calls = 0;
inline bool next_wait_fails = false;  // the next wait for a stream says that something on it went wrong

inline bool fails() { return calls++ == fail_at; }
inline bool inside(const std::map<const char*, size_t>& m, const void* p, size_t bytes) {
    auto it = m.upper_bound((const char*)p);
    if (it == m.begin()) return false;
    --it;
    return (const char*)p + bytes <= it->first + it->second;
}
inline bool overlap(const void* a, size_t na, const void* b, size_t nb) { return (const char*)a < (const char*)b + nb && (const char*)b < (const char*)a + na; }
inline void run(Stream* s, unsigned long long upto) {
    while (s->done < upto) {
        Op op = s->q.front();
        s->q.pop_front();
        s->done++;
        if (op.wait) {
            if (op.wait->s) run(op.wait->s, op.upto);
            continue;
        }
        const char* from = op.held.empty() ? op.from : op.held.data();
        const bool to_ok = inside(device, op.to, op.bytes) || inside(locked, op.to, op.bytes);
        const bool from_ok = !op.held.empty() || inside(device, from, op.bytes) || inside(locked, from, op.bytes);
        if (!to_ok || !from_ok) { faults.push_back("a copy to or from memory that is gone"); continue; }
        memcpy(op.to, from, op.bytes);
    }
}
// whether work that is still to be done touches these bytes
inline bool busy(const void* p, size_t bytes, const Stream* but = nullptr) {
    for (Stream* s : streams) {
        if (s == but) continue;
        for (auto& op : s->q)
            if (!op.wait && (overlap(op.to, op.bytes, p, bytes) || (op.held.empty() && overlap(op.from, op.bytes, p, bytes)))) return true;
    }
    return false;
}

}  // namespace fake

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof *p);
    strcpy(p->name, "none");
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    fake::streams.push_back(new fake::Stream());
    *s = (cudaStream_t)fake::streams.back();
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    fake::run((fake::Stream*)s, ((fake::Stream*)s)->issued);
    const bool bad = fake::next_wait_fails;
    fake::next_wait_fails = false;
    return bad ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    for (auto it = fake::streams.begin(); it != fake::streams.end(); ++it)
        if (*it == (fake::Stream*)s) { fake::streams.erase(it); break; }
    delete (fake::Stream*)s;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { if (fake::fails()) return cudaErrorMemoryAllocation; *e = (cudaEvent_t) new fake::Event(); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (fake::Event*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (fake::fails()) return cudaErrorUnknown;
    ((fake::Event*)e)->s = (fake::Stream*)s;
    ((fake::Event*)e)->seq = ((fake::Stream*)s)->issued;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    fake::Event* v = (fake::Event*)e;
    if (!v->s || v->s->done >= v->seq) return cudaSuccess;
    fake::run(v->s, v->s->done + 1);  // the device gets on a little
    return cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    fake::Event* v = (fake::Event*)e;
    if (v->s) fake::run(v->s, v->seq);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (fake::fails()) return cudaErrorUnknown;
    fake::Event* v = (fake::Event*)e;
    if (!v->s) return cudaSuccess;
    // by value: the event may be recorded again before the wait is reached
    fake::Event* at = new fake::Event(*v);
    ((fake::Stream*)s)->q.push_back({nullptr, nullptr, 0, {}, at, at->seq});
    ((fake::Stream*)s)->issued++;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = calloc(1, n);
    fake::device[(const char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { fake::device.erase((const char*)p); free(p); return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return fake::fails() ? cudaErrorMemoryAllocation : cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
    fake::run((fake::Stream*)s, ((fake::Stream*)s)->issued);
    if (fake::busy(p, fake::device[(const char*)p])) fake::faults.push_back("device memory freed under a copy on another stream");
    return cudaFree(p);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (fake::fails()) return cudaErrorMemoryAllocation;
    *p = calloc(1, n);
    fake::locked[(const char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    if (fake::busy(p, fake::locked[(const char*)p])) fake::faults.push_back("page-locked memory freed under a copy");
    fake::locked.erase((const char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    memset(a, 0, sizeof *a);
    a->type = fake::inside(fake::locked, p, 1) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    if (fake::fails()) return cudaErrorUnknown;
    fake::Stream* s = (fake::Stream*)st;
    fake::Op op{(char*)to, (const char*)from, n, {}, nullptr, 0};
    // pageable memory: an upload takes the bytes along at once, a download waits
    if (kind == cudaMemcpyHostToDevice && !fake::inside(fake::locked, from, n)) op.held.assign((const char*)from, (const char*)from + n);
    if (kind == cudaMemcpyDeviceToHost && !fake::inside(fake::locked, to, n)) {
        fake::run(s, s->issued);
        memcpy(to, from, n);
        return cudaSuccess;
    }
    s->q.push_back(op);
    s->issued++;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { if (fake::fails()) return cudaErrorUnknown; memset(p, v, n); return cudaSuccess; }
}
