// Runs the blocks of a CUDA kernel on the CPU, one block at a time, for checks
// that no GPU run can make safely or at will: every thread is a fiber, and the
// fibers take turns in the order of their index from one synchronisation to
// the next.  Covers what the kernels under test use: shared memory, block
// barriers, warp votes and shuffles, atomics.  The kernel's source is compiled as
// C++ after this header (launches replaced).
#pragma once
#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <vector>

#undef __shared__
#define __shared__ static
#undef __launch_bounds__
#define __launch_bounds__(...)

namespace host_block {

struct Block {
    uint32_t size = 0, current = 0;
    ucontext_t scheduler{};
    std::vector<ucontext_t> context;
    std::vector<std::vector<char>> stack;
    std::vector<char> done, waiting;   // waiting: at a block barrier
    // warp collectives: two slots per warp, used in turn
    struct Slot {
        uint64_t value[32];
        uint32_t arrived, turn;
    };
    std::vector<Slot> slots;
    std::vector<uint32_t> turn;        // collectives entered, per thread
    std::function<void()> body;
    bool left = false;                 // a thread returned while others went on to a barrier
};
inline Block* block = nullptr;

inline void yield() { swapcontext(&block->context[block->current], &block->scheduler); }

inline uint32_t lanes_alive() {
    const uint32_t w = block->current / 32u;
    uint32_t m = 0;
    for (uint32_t l = 0; l < 32u && 32u * w + l < block->size; l++)
        if (!block->done[32u * w + l]) m |= 1u << l;
    return m;
}

// Deposits v and returns the slot once every live lane of the warp has.
inline const Block::Slot& exchange(uint64_t v) {
    const uint32_t t = block->current, turn = block->turn[t]++;
    Block::Slot& s = block->slots[2u * (t / 32u) + (turn & 1u)];
    if (s.turn != turn + 1u) {
        s.turn = turn + 1u;
        s.arrived = 0u;
    }
    s.value[t % 32u] = v;
    s.arrived |= 1u << (t % 32u);
    while ((s.arrived & lanes_alive()) != lanes_alive()) yield();
    return s;
}

inline void entry() {
    Block* b = block;
    b->body();
    b->done[b->current] = 1;
    swapcontext(&b->context[b->current], &b->scheduler);
}

// One block of `size` threads; after(t) is called whenever thread t has run to
// its next synchronisation.  False when a thread had returned before a block
// barrier that others waited at, or when no thread can go on.
inline bool run(uint32_t size, const std::function<void()>& body,
                const std::function<void(uint32_t)>& after = {}) {
    Block b;
    b.size = size;
    b.context.resize(size);
    b.stack.assign(size, std::vector<char>(128 << 10));
    b.done.assign(size, 0);
    b.waiting.assign(size, 0);
    b.slots.resize(2 * ((size + 31) / 32));
    for (auto& s : b.slots) s.arrived = s.turn = 0;
    b.turn.assign(size, 0);
    b.body = body;
    block = &b;
    for (uint32_t t = 0; t < size; t++) {
        getcontext(&b.context[t]);
        b.context[t].uc_stack.ss_sp = b.stack[t].data();
        b.context[t].uc_stack.ss_size = b.stack[t].size();
        b.context[t].uc_link = &b.scheduler;
        makecontext(&b.context[t], entry, 0);
    }
    for (uint64_t idle = 0; idle < 1000000;) {
        bool moved = false;
        uint32_t live = 0, waiting = 0;
        for (uint32_t t = 0; t < size; t++) {
            if (!b.done[t] && !b.waiting[t]) {
                b.current = t;
                swapcontext(&b.scheduler, &b.context[t]);
                if (after) after(t);
                moved = true;
            }
            live += b.done[t] ? 0u : 1u;
            waiting += (!b.done[t] && b.waiting[t]) ? 1u : 0u;
        }
        if (live == 0) return !b.left;
        if (waiting == live) {
            if (live != size) b.left = true;
            std::fill(b.waiting.begin(), b.waiting.end(), char(0));
        }
        idle = moved ? idle + 1 : idle + 100000;
    }
    return false;
}

}  // namespace host_block

// ---- what the kernels call ---------------------------------------------------
struct HostIndex {
    struct Thread {
        operator uint32_t() const { return host_block::block->current; }
    } x;
};
static HostIndex threadIdx;
static uint3 blockIdx;
static dim3 blockDim, gridDim;

inline void __syncthreads() {
    host_block::block->waiting[host_block::block->current] = 1;
    host_block::yield();
}
inline uint32_t __ballot_sync(uint32_t, bool p) {
    const auto& s = host_block::exchange(p ? 1u : 0u);
    uint32_t m = 0;
    for (uint32_t l = 0; l < 32u; l++)
        if (((s.arrived >> l) & 1u) && s.value[l]) m |= 1u << l;
    return m;
}
template <class T>
inline T host_shuffle(T v, int from) {
    uint64_t bits = 0;
    std::memcpy(&bits, &v, sizeof(T));
    const auto& s = host_block::exchange(bits);
    T r;
    std::memcpy(&r, &s.value[from & 31], sizeof(T));
    return r;
}
template <class T>
inline T __shfl_xor_sync(uint32_t, T v, int o) {
    return host_shuffle(v, int(threadIdx.x % 32u) ^ o);
}
template <class T>
inline T __shfl_up_sync(uint32_t, T v, int o) {
    const int lane = int(threadIdx.x % 32u);
    return host_shuffle(v, lane >= o ? lane - o : lane);
}
template <class T, class U>
inline T atomicAdd(T* p, U v) {
    const T old = *p;
    *p = T(old + T(v));
    return old;
}
inline uint32_t atomicExch(uint32_t* p, uint32_t v) {
    const uint32_t old = *p;
    *p = v;
    return old;
}
inline int __ffs(int v) { return __builtin_ffs(v); }
template <class T, class F>
inline T host_bits(F f) {
    T t;
    std::memcpy(&t, &f, 4);
    return t;
}
inline uint32_t __float_as_uint(float f) { return host_bits<uint32_t>(f); }
inline int __float_as_int(float f) { return host_bits<int>(f); }
inline float __uint_as_float(uint32_t u) { return host_bits<float>(u); }
inline float __int_as_float(int i) { return host_bits<float>(i); }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return uint32_t((uint64_t(a) * b) >> 32); }
using std::max;
using std::min;
inline void host_no_launch(...) {}

namespace mrb {
void set_error(const char*, ...) {}
}  // namespace mrb
