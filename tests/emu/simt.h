// simt.h -- TEST INFRASTRUCTURE: runs CUDA device code of one thread block on the host.
//
// Every thread is a fiber that runs until its next warp- or block-wide operation
// (__syncwarp, __shfl_xor_sync, __syncthreads); the operation completes when all
// threads of the warp or block have reached the same one.  A block in which that
// cannot happen (threads at different operations, or finished ones) is reported, as
// is a shuffle whose lanes are not all there.  Asynchronous copies land when the
// copying thread waits for them, not before.
#pragma once
#include <setjmp.h>
#include <string.h>
#include <ucontext.h>

#include <cmath>
#include <functional>
#include <stdexcept>
#include <utility>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) __attribute__((aligned(n)))

struct int2 {
    int x, y;
};
inline int2 make_int2(int x, int y) { return int2{x, y}; }
struct Dim {
    int x = 0, y = 0, z = 0;
};

namespace simt {

enum class At { Ready, Warp, Block, Done };

struct Thread {
    ucontext_t ctx;
    jmp_buf jb;
    std::vector<char> stack;
    At at = At::Ready;
    int op = 0;        // kind of the operation it waits at
    unsigned turn = 0; // warp operations so far
    std::vector<std::pair<double *, const double *>> copies;  // 16 bytes each
};

struct Machine {
    std::vector<Thread> threads;
    std::vector<double> slots;  // [warp][2][lane]: shuffled values
    jmp_buf sched;
    int now = 0;
    std::function<void()> body;
    const char *fault = nullptr;
};
inline Machine &machine() {
    static thread_local Machine m;
    return m;
}

inline void wait_at(At at, int op) {
    Machine &m = machine();
    Thread &t = m.threads[m.now];
    t.at = at;
    t.op = op;
    if (!_setjmp(t.jb)) _longjmp(m.sched, 1);
}

inline void entry() {
    Machine &m = machine();
    m.body();
    m.threads[m.now].at = At::Done;
    _longjmp(m.sched, 1);
}

}  // namespace simt

inline thread_local Dim threadIdx, blockIdx, blockDim, gridDim;

namespace simt {

inline void resume(Thread &t, int i, bool first) {
    Machine &m = machine();
    m.now = i;
    threadIdx.x = i;
    t.at = At::Ready;
    if (_setjmp(m.sched)) return;
    if (first) setcontext(&t.ctx);
    else _longjmp(t.jb, 1);
}

// Run body as a block of n threads (a multiple of 32).
inline void run_block(int n, std::function<void()> body) {
    Machine &m = machine();
    m.body = std::move(body);
    m.fault = nullptr;
    if ((int)m.threads.size() < n) m.threads.resize(n);
    m.slots.assign((size_t)n * 2, 0.0);
    blockDim.x = n;
    std::vector<char> started(n, 0);
    for (int i = 0; i < n; ++i) {
        Thread &t = m.threads[i];
        if (t.stack.empty()) t.stack.resize(256 << 10);
        t.at = At::Ready;
        t.turn = 0;
        t.copies.clear();
        getcontext(&t.ctx);
        t.ctx.uc_stack.ss_sp = t.stack.data();
        t.ctx.uc_stack.ss_size = t.stack.size();
        t.ctx.uc_link = nullptr;
        makecontext(&t.ctx, entry, 0);
    }
    for (;;) {
        for (int w = 0; w < n; w += 32)
            for (;;) {
                for (int i = w; i < w + 32; ++i)
                    if (m.threads[i].at == At::Ready) {
                        resume(m.threads[i], i, !started[i]);
                        started[i] = 1;
                    }
                int at_warp = 0;
                for (int i = w; i < w + 32; ++i)
                    at_warp += m.threads[i].at == At::Warp && m.threads[i].op == m.threads[w].op && m.threads[i].turn == m.threads[w].turn;
                bool any = false;
                for (int i = w; i < w + 32; ++i) any = any || m.threads[i].at == At::Warp;
                if (!any) break;
                if (at_warp < 32) throw std::runtime_error("simt: a warp-wide operation that some lanes do not reach");
                for (int i = w; i < w + 32; ++i) m.threads[i].at = At::Ready;
            }
        int block = 0, done = 0;
        for (int i = 0; i < n; ++i) {
            block += m.threads[i].at == At::Block;
            done += m.threads[i].at == At::Done;
        }
        if (done == n) break;
        if (block < n) throw std::runtime_error("simt: a block barrier that some threads do not reach");
        for (int i = 0; i < n; ++i) m.threads[i].at = At::Ready;
    }
    for (int i = 0; i < n; ++i)
        if (!m.threads[i].copies.empty()) throw std::runtime_error("simt: a copy that nobody waited for");
}

// 16 bytes, visible after this thread's copies_wait
inline void copy16(double *dst, const double *src) {
    if (((size_t)dst | (size_t)src) & 15) throw std::runtime_error("simt: misaligned 16-byte copy");
    machine().threads[machine().now].copies.push_back({dst, src});
}
inline void copies_wait() {
    auto &c = machine().threads[machine().now].copies;
    for (auto &p : c) memcpy(p.first, p.second, 16);
    c.clear();
}

}  // namespace simt

inline void __syncwarp() {
    ++simt::machine().threads[simt::machine().now].turn;
    simt::wait_at(simt::At::Warp, 1);
}
inline void __syncthreads() { simt::wait_at(simt::At::Block, 2); }
inline double __shfl_xor_sync(unsigned, double v, int o) {
    simt::Machine &m = simt::machine();
    const int i = m.now;
    const unsigned par = ++m.threads[i].turn & 1;
    const size_t base = (size_t)(i & ~31) * 2 + par * 32;
    m.slots[base + (i & 31)] = v;
    simt::wait_at(simt::At::Warp, 16 + o);
    return simt::machine().slots[base + ((i & 31) ^ o)];
}
inline int atomicOr(int *p, int v) {
    const int o = *p;
    *p |= v;
    return o;
}
inline int atomicMin(int *p, int v) {
    const int o = *p;
    if (v < o) *p = v;
    return o;
}
using std::isfinite;
inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
