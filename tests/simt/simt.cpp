// The stand-in's fibers, streams and allocations (cuda_runtime.h in this folder).
#include "cuda_runtime.h"

#include <ucontext.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>
#include <memory>
#include <string>
#include <vector>

namespace simt {

Thread* self = nullptr;
Dim block_idx, grid_dim, block_dim;

namespace {

enum State { kReady, kWarp, kBlock, kNamed, kDone };
constexpr size_t kStack = 256 << 10;
struct Fiber : Thread {
    ucontext_t ctx;
    std::unique_ptr<char[]> stack{new char[kStack]};
    State state;
    int line, id, p;
    unsigned gen;
};
struct Warp {
    unsigned arrived, gen;
    int line;
    uint64_t slot[2][32];
};
std::vector<std::unique_ptr<Fiber>> pool;
std::vector<Warp> warps;
ucontext_t scheduler;
std::function<void()>* body;
int barrier_sum;
alignas(16) unsigned char shared_memory[228 << 10];

std::string fault, current, drop;
std::map<std::string, uint64_t> barriers;  // of each kernel since simt_clear
long long barrier_clock = 0;
int order = 0;

void flag(const std::string& what) {
    if (fault.empty()) fault = current + ": " + what;
}
Fiber* me() { return static_cast<Fiber*>(self); }
void yield() {
    Fiber* f = me();
    swapcontext(&f->ctx, &scheduler);
}
void entry() {
    (*body)();
    me()->state = kDone;
    yield();
}

// Runs the block to its end; false when its threads wait for one another in vain.
bool run_block(unsigned n) {
    const unsigned nw = (n + 31) / 32;
    warps.assign(nw, Warp{});
    for (unsigned i = 0; i < n; ++i) {
        if (pool.size() <= i) pool.push_back(std::make_unique<Fiber>());
        Fiber* f = pool[i].get();
        f->tid = Dim{i, 0, 0};
        f->state = kReady;
        f->gen = 0;
        getcontext(&f->ctx);
        f->ctx.uc_stack.ss_sp = f->stack.get();
        f->ctx.uc_stack.ss_size = kStack;
        f->ctx.uc_link = nullptr;
        makecontext(&f->ctx, entry, 0);
    }
    for (;;) {
        for (unsigned k = 0; k < nw; ++k) {
            const unsigned w = order & 1 ? nw - 1 - k : k, first = 32 * w, lanes = std::min(n - first, 32u);
            for (bool again = true; again;) {
                again = false;
                for (unsigned l = 0; l < lanes; ++l) {
                    Fiber* f = pool[first + (order & 2 ? lanes - 1 - l : l)].get();
                    if (f->state == kWarp && f->gen != warps[w].gen) f->state = kReady;
                    if (f->state != kReady) continue;
                    self = f;
                    swapcontext(&scheduler, &f->ctx);
                    again = true;
                }
            }
        }
        unsigned at[5] = {0, 0, 0, 0, 0};
        int line = -1, id = -1, count = 0;
        bool mixed = false;
        barrier_sum = 0;
        for (unsigned i = 0; i < n; ++i) {
            Fiber* f = pool[i].get();
            ++at[f->state];
            if (f->state == kBlock) {
                mixed |= line >= 0 && line != f->line;
                line = f->line;
                barrier_sum += f->p;
            }
            if (f->state == kNamed) {
                id = f->id;
                count = f->p;
            }
        }
        if (at[kDone] == n) return true;
        if (id >= 0 && (int)at[kNamed] == count) {
            for (unsigned i = 0; i < n; ++i)
                if (pool[i]->state == kNamed) pool[i]->state = kReady;
            continue;
        }
        if (at[kBlock] == n && !mixed) {
            ++barriers[current];
            barrier_clock += 4096;
            for (unsigned i = 0; i < n; ++i) pool[i]->state = kReady;
            continue;
        }
        flag("threads of one block wait at different places (line " + std::to_string(line) + ": " +
             std::to_string(at[kBlock]) + " of " + std::to_string(n) + ", ended: " + std::to_string(at[kDone]) +
             ", at a warp collective: " + std::to_string(at[kWarp]) + (mixed ? ", several barriers" : "") + ")");
        return false;
    }
}

}  // namespace

void barrier(int line) {
    Fiber* f = me();
    f->state = kBlock;
    f->line = line;
    f->p = 0;
    yield();
}
int barrier_count(int line, int p) {
    Fiber* f = me();
    f->state = kBlock;
    f->line = line;
    f->p = p != 0;
    yield();
    return barrier_sum;
}
void named_barrier(int id, int count) {
    Fiber* f = me();
    f->state = kNamed;
    f->id = id;
    f->p = count;
    yield();
}
const uint64_t* exchange(int line, uint64_t v) {
    Fiber* f = me();
    Warp& w = warps[f->tid.x / 32];
    const unsigned gen = w.gen;
    if (w.arrived && w.line != line) flag("lanes of one warp at lines " + std::to_string(w.line) + " and " + std::to_string(line));
    w.line = line;
    w.slot[gen & 1][f->tid.x & 31] = v;
    if (++w.arrived == 32 || (block_dim.x < 32 && w.arrived == block_dim.x)) {
        w.arrived = 0;
        ++w.gen;
    } else {
        f->state = kWarp;
        f->gen = gen;
        yield();
    }
    return w.slot[gen & 1];
}
long long ticks() { return barrier_clock; }
void* dynamic_shared() { return shared_memory; }
bool dropped() { return !drop.empty() && current.find(drop) != std::string::npos; }

// ---------------------------------------------------------------- streams -----------------
namespace {
struct Stream {
    std::deque<std::function<void()>> ops;
    uint64_t done = 0, issued = 0;
};
struct Event {
    Stream* stream = nullptr;
    uint64_t seq = 0;
};
Stream null_stream;
std::map<Stream*, int> streams{{&null_stream, 0}};
struct Region {
    size_t bytes;
    bool pinned;          // host memory
    int device = 0;
    char* data = nullptr; // another device's memory: what copies read; kernels find poison at its address
};
std::map<const char*, Region> memory;
size_t malloc_limit = ~size_t(0);
std::string kernels;

Stream* of(cudaStream_t s) { return s ? reinterpret_cast<Stream*>(s) : &null_stream; }
void run_to(Stream* s, uint64_t seq) {
    while (s->done < seq) {
        auto op = std::move(s->ops.front());
        s->ops.pop_front();
        ++s->done;
        op();
    }
}
void issue(cudaStream_t s, std::function<void()> op) {
    of(s)->ops.push_back(std::move(op));
    ++of(s)->issued;
}
void run_all() {
    for (auto& s : streams) run_to(s.first, s.first->issued);
}
const std::pair<const char* const, Region>* find(const void* p) {
    auto it = memory.upper_bound(static_cast<const char*>(p));
    if (it == memory.begin()) return nullptr;
    --it;
    return static_cast<const char*>(p) < it->first + it->second.bytes ? &*it : nullptr;
}
bool pageable(const void* p) { return !find(p); }
const void* readable(const void* p) {
    auto* m = find(p);
    return m && m->second.data ? m->second.data + (static_cast<const char*>(p) - m->first) : p;
}
void* take(size_t n, bool pinned, unsigned char poison) {
    void* p = nullptr;  // (to the next 16 bytes, no further: an address sanitizer sees what reads or writes beyond)
    if (posix_memalign(&p, 256, (n + 15) / 16 * 16)) return nullptr;
    std::memset(p, poison, n);
    memory[static_cast<char*>(p)] = Region{n, pinned};
    return p;
}
}  // namespace

void queue(const char* name, Config c, std::function<void()> kernel) {
    kernels += std::string(name) + "\n";
    issue(c.stream, [=]() mutable {
        current = name;
        grid_dim = Dim{c.grid, 1, 1};
        block_dim = Dim{c.block, 1, 1};
        body = &kernel;
        for (unsigned b = 0; b < c.grid; ++b) {
            block_idx = Dim{b, 0, 0};
            std::memset(shared_memory, 0xA7, c.smem);
            if (!run_block(c.block)) return;
        }
    });
}

}  // namespace simt

using namespace simt;

cudaError_t simt_malloc(void** p, size_t n) {
    *p = nullptr;
    if (n > malloc_limit) return cudaErrorMemoryAllocation;
    *p = take(n, false, 0xA5);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    run_all();
    memory.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = take(n, true, 0x5A);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    if (k == cudaMemcpyHostToDevice && pageable(s)) {
        auto copy = std::make_shared<std::vector<char>>(static_cast<const char*>(s), static_cast<const char*>(s) + n);
        issue(st, [=] { std::memcpy(d, copy->data(), n); });
    } else {
        if (k == cudaMemcpyDeviceToDevice && (pageable(d) || pageable(s))) return cudaErrorInvalidValue;
        issue(st, [=] { std::memmove(d, readable(s), n); });
        if (k == cudaMemcpyDeviceToHost && pageable(d)) return cudaStreamSynchronize(st);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    run_to(&null_stream, null_stream.issued);
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    issue(st, [=] { std::memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    run_to(&null_stream, null_stream.issued);
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    auto* n = new Stream;
    streams[n] = 0;
    *s = reinterpret_cast<cudaStream_t>(n);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    run_to(of(s), of(s)->issued);
    streams.erase(of(s));  // (kept for events that still name it)
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    run_to(of(s), of(s)->issued);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    const Event ev = *reinterpret_cast<Event*>(e);
    issue(s, [=] {
        if (ev.stream) run_to(ev.stream, ev.seq);
    });
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete reinterpret_cast<Event*>(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    *reinterpret_cast<Event*>(e) = Event{of(s), of(s)->issued};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    const Event ev = *reinterpret_cast<Event*>(e);
    if (ev.stream) run_to(ev.stream, ev.seq);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : e ? "invalid argument" : "no error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceReset() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    *a = cudaPointerAttributes{};
    if (auto* m = find(p)) {
        a->type = m->second.pinned ? cudaMemoryTypeHost : cudaMemoryTypeDevice;
        a->device = m->second.device;
    }
    return cudaSuccess;
}

extern "C" {
void simt_order(int o) { order = o; }  // bit 0: the last warp first; bit 1: the last lane first
const char* simt_fault() { return fault.c_str(); }
void simt_clear() {
    fault.clear();
    kernels.clear();
    barriers.clear();
}
const char* simt_kernels() { return kernels.c_str(); }  // launched, one per line
// Barriers that the kernels of this name have met, over all their blocks.
uint64_t simt_barriers(const char* name) {
    uint64_t n = 0;
    for (auto& b : barriers)
        if (b.first.find(name) != std::string::npos) n += b.second;
    return n;
}
// Work that has been queued and not run.
uint64_t simt_pending() {
    uint64_t n = 0;
    for (auto& s : streams) n += s.first->ops.size();
    return n;
}
void simt_malloc_limit(uint64_t n) { malloc_limit = n; }
void simt_drop_status(const char* kernel) { drop = kernel; }
void* simt_device_alloc(uint64_t n) { return take(n, false, 0xA5); }
void* simt_pinned_alloc(uint64_t n) { return take(n, true, 0x5A); }
// Another device's memory, which only copies reach; *data is where its contents are.
void* simt_peer_alloc(uint64_t n, void** data) {
    char* p = static_cast<char*>(take(n, false, 0xD1));
    memory[p].device = 1;
    *data = memory[p].data = static_cast<char*>(std::malloc(n));
    return p;
}
void simt_device_free(void* p) {  // at once, without waiting for queued work
    memory.erase(static_cast<char*>(p));
    std::free(p);
}
}
