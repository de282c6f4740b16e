/*
 * cuda_runtime.h -- lets the Tier-1 kernels' device code compile as host C++
 * and run one warp at a time on the CPU (TEST INFRASTRUCTURE ONLY).
 *
 * Each lane is a fiber.  A lane runs alone, without interruption, until it
 * reaches a warp barrier, shuffle or vote, and the lanes take their turns in
 * an order that the test chooses.  So between two synchronisation points some
 * lane always runs as far ahead of the others as the programming model lets
 * it: code that counts on lanes staying together without a barrier reads
 * another lane's later value here.  Lanes that wait for one another at
 * different synchronisation points, or that leave while others wait, are
 * reported instead of hanging.
 */
#pragma once

#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __constant__ static const
#define __shared__ static
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __align__(n) alignas(n)
#define __launch_bounds__(...)

using std::max;
using std::min;

struct uint2 {
    uint32_t x, y;
};
inline uint2 make_uint2(uint32_t x, uint32_t y) { return uint2{x, y}; }

namespace emu {

struct Dim {
    unsigned x = 0;
};

struct Lane {
    ucontext_t at;
    std::vector<char> stack;
    bool waiting = false, done = false;
    unsigned mask = 0;    // lanes it waits for
    int kind = 0;         // the kind of synchronisation point it waits at
    uint64_t value = 0;   // what it brings there
    uint64_t seen[32];    // what the lanes brought to the last one
};

struct Warp {
    Lane lane[32];
    ucontext_t home;
    int current = 0;
    std::function<void(int)> body;
};
inline Warp *&warp()
{
    static Warp *w = nullptr;
    return w;
}

inline void entry()
{
    Warp &w = *warp();
    const int l = w.current;
    w.body(l);
    w.lane[l].done = true;
    swapcontext(&w.lane[l].at, &w.home);
}

// Waits for the lanes of mask; returns what each of them brought.
inline const uint64_t *meet(unsigned mask, int kind, uint64_t value)
{
    Warp &w = *warp();
    Lane &me = w.lane[w.current];
    me.waiting = true;
    me.mask = mask;
    me.kind = kind;
    me.value = value;
    swapcontext(&me.at, &w.home);
    return me.seen;
}

// Runs body(lane) on 32 lanes, taken in `order`; false if they got stuck.
inline bool run(const int (&order)[32], std::function<void(int)> body)
{
    static Warp w;
    warp() = &w;
    w.body = std::move(body);
    for (int l = 0; l < 32; l++) {
        Lane &L = w.lane[l];
        L.stack.resize(256 * 1024);
        L.waiting = L.done = false;
        getcontext(&L.at);
        L.at.uc_stack.ss_sp = L.stack.data();
        L.at.uc_stack.ss_size = L.stack.size();
        L.at.uc_link = nullptr;
        makecontext(&L.at, entry, 0);
    }
    for (;;) {
        bool progress = false, all_done = true;
        for (int i = 0; i < 32; i++) {
            Lane &L = w.lane[order[i]];
            if (L.done) continue;
            all_done = false;
            if (L.waiting) {
                // does everyone that it waits for wait for the same?
                bool ready = true;
                for (int k = 0; k < 32; k++) {
                    if (!((L.mask >> k) & 1u)) continue;
                    const Lane &K = w.lane[k];
                    if (!K.waiting || K.mask != L.mask || K.kind != L.kind) ready = false;
                }
                if (!ready) continue;
                for (int k = 0; k < 32; k++) {
                    if (!((L.mask >> k) & 1u)) continue;
                    for (int j = 0; j < 32; j++) w.lane[k].seen[j] = w.lane[j].value;
                    w.lane[k].waiting = false;
                }
            }
            progress = true;
            w.current = order[i];
            swapcontext(&w.home, &L.at);
        }
        if (all_done) return true;
        if (!progress) return false;
    }
}

template <typename T>
uint64_t bits_of(T v)
{
    uint64_t b = 0;
    std::memcpy(&b, &v, sizeof v);
    return b;
}
template <typename T>
T value_of(uint64_t b)
{
    T v;
    std::memcpy(&v, &b, sizeof v);
    return v;
}

}  // namespace emu

namespace emu {
inline Dim thread_idx() { return Dim{(unsigned)warp()->current}; }
static Dim block_idx;
constexpr Dim kBlockDim{32};
}  // namespace emu
#define threadIdx (emu::thread_idx())
#define blockIdx (emu::block_idx)
#define blockDim (emu::kBlockDim)

inline void __syncthreads() { emu::meet(0xffffffffu, 0, 0); }
inline void __syncwarp(unsigned mask = 0xffffffffu) { emu::meet(mask, 1, 0); }
template <typename T>
T __shfl_sync(unsigned mask, T v, int src)
{
    return emu::value_of<T>(emu::meet(mask, 2, emu::bits_of(v))[src & 31]);
}
template <typename T>
T __shfl_up_sync(unsigned mask, T v, unsigned d)
{
    const int l = emu::warp()->current, s = l - (int)d;
    return emu::value_of<T>(emu::meet(mask, 3, emu::bits_of(v))[s < 0 ? l : s]);
}
template <typename T>
T __shfl_down_sync(unsigned mask, T v, unsigned d)
{
    const int l = emu::warp()->current, s = l + (int)d;
    return emu::value_of<T>(emu::meet(mask, 4, emu::bits_of(v))[s > 31 ? l : s]);
}
template <typename T>
T __shfl_xor_sync(unsigned mask, T v, int x)
{
    const int l = emu::warp()->current;
    return emu::value_of<T>(emu::meet(mask, 5, emu::bits_of(v))[l ^ x]);
}
inline unsigned __ballot_sync(unsigned mask, bool p)
{
    const uint64_t *s = emu::meet(mask, 6, p);
    unsigned b = 0;
    for (int k = 0; k < 32; k++) b |= ((mask >> k) & 1u) && s[k] ? 1u << k : 0u;
    return b;
}
inline bool __any_sync(unsigned mask, bool p) { return __ballot_sync(mask, p) != 0u; }

inline void __threadfence() {}
template <typename T>
T __ldg(const T *p)
{
    return *p;
}
template <typename T>
T __ldcg(const T *p)
{
    return *p;
}
inline uint32_t atomicOr(uint32_t *p, uint32_t v)
{
    const uint32_t o = *p;
    *p |= v;
    return o;
}
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s)
{
    return (uint32_t)((((uint64_t)hi << 32 | lo) << (s & 31)) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s)
{
    return (uint32_t)(((uint64_t)hi << 32 | lo) >> (s & 31));
}
inline uint32_t __float_as_uint(float f) { return emu::value_of<uint32_t>(emu::bits_of(f)); }
inline float __uint_as_float(uint32_t u) { return emu::value_of<float>(u); }
