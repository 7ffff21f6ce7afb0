// Host stand-ins for what the kernels use of the device: a thread of a block
// is a host thread.  __syncwarp and __syncthreads order memory; shuffles,
// votes and reductions bring their lanes together and exchange values but
// order nothing, as PTX has it.  Under ThreadSanitizer a missing barrier
// between two accesses of shared memory is then a reported data race.
#pragma once
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <sched.h>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#undef __launch_bounds__
#define __launch_bounds__(...)

struct Dim { unsigned x = 0, y = 0, z = 0; };
inline thread_local Dim threadIdx, blockIdx;
inline Dim blockDim;
alignas(64) inline unsigned char dynamic_smem[1 << 18];

// A meeting point of n threads; kOrder: memory before it is visible after it.
struct Meet {
    std::atomic<int> in{0}, generation{0};
    std::atomic<uint64_t> slot[2][32];
    template <bool kOrder>
    void wait(int n)
    {
        constexpr auto arrive = kOrder ? std::memory_order_acq_rel : std::memory_order_relaxed;
        constexpr auto leave = kOrder ? std::memory_order_acquire : std::memory_order_relaxed;
        const int g = generation.load(std::memory_order_relaxed);
        if (in.fetch_add(1, arrive) == n - 1) {
            in.store(0, std::memory_order_relaxed);
            generation.fetch_add(1, arrive);
        } else {
            while (generation.load(leave) == g) sched_yield();
        }
    }
};
inline Meet warps[16], whole_block;
inline thread_local int parity = 0;
inline int lane() { return static_cast<int>(threadIdx.x & 31); }
inline void __syncwarp(unsigned = ~0u) { warps[threadIdx.x >> 5].wait<true>(32); }
inline void __syncthreads() { whole_block.wait<true>(static_cast<int>(blockDim.x)); }

template <typename To, typename From>
To recast(From v)
{
    uint64_t bits = 0;
    std::memcpy(&bits, &v, sizeof(From));
    To r;
    std::memcpy(&r, &bits, sizeof(To));
    return r;
}
// The values of the warp's lanes.
struct Lanes {
    uint64_t v[32];
    explicit Lanes(uint64_t mine)
    {
        Meet &m = warps[threadIdx.x >> 5];
        auto &s = m.slot[parity];
        parity ^= 1;
        s[lane()].store(mine, std::memory_order_relaxed);
        m.wait<false>(32);
        for (int i = 0; i < 32; ++i) v[i] = s[i].load(std::memory_order_relaxed);
    }
};
template <typename T> T __shfl_sync(unsigned, T v, int src, int w = 32)
{
    return recast<T>(Lanes(recast<uint64_t>(v)).v[(lane() & ~(w - 1)) | (src & (w - 1))]);
}
template <typename T> T __shfl_up_sync(unsigned, T v, int d, int w = 32)
{
    return recast<T>(Lanes(recast<uint64_t>(v)).v[(lane() & (w - 1)) >= d ? lane() - d : lane()]);
}
template <typename T> T __shfl_xor_sync(unsigned, T v, int d, int = 32)
{
    return recast<T>(Lanes(recast<uint64_t>(v)).v[lane() ^ d]);
}
inline unsigned __ballot_sync(unsigned, int p)
{
    const Lanes all(p != 0);
    unsigned b = 0;
    for (int i = 0; i < 32; ++i) b |= static_cast<unsigned>(all.v[i]) << i;
    return b;
}
inline int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
inline unsigned __reduce_max_sync(unsigned, unsigned v)
{
    const Lanes all(v);
    return static_cast<unsigned>(*std::max_element(all.v, all.v + 32));
}
inline int __reduce_min_sync(unsigned, int v)      // (of values >= 0)
{
    const Lanes all(static_cast<unsigned>(v));
    return static_cast<int>(*std::min_element(all.v, all.v + 32));
}

using std::max;
using std::min;
inline unsigned max(unsigned a, int b) { return std::max(a, static_cast<unsigned>(b)); }
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __ffs(unsigned x) { return __builtin_ffs(static_cast<int>(x)); }
inline int __clz(int x) { return x ? __builtin_clz(static_cast<unsigned>(x)) : 32; }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return static_cast<uint32_t>((static_cast<uint64_t>(a) * b) >> 32); }
inline uint64_t __umul64hi(uint64_t a, uint64_t b)
{
    return static_cast<uint64_t>((static_cast<unsigned __int128>(a) * b) >> 64);
}
inline uint32_t __float_as_uint(float f) { return recast<uint32_t>(f); }
inline int __float_as_int(float f) { return recast<int>(f); }
inline float __int_as_float(int i) { return recast<float>(i); }
inline float __uint_as_float(uint32_t i) { return recast<float>(i); }
inline long long __double_as_longlong(double d) { return recast<long long>(d); }
inline int __double2hiint(double d) { return static_cast<int>(recast<uint64_t>(d) >> 32); }
inline int __double2loint(double d) { return static_cast<int>(recast<uint64_t>(d)); }
inline double __hiloint2double(int h, int l)
{
    return recast<double>((static_cast<uint64_t>(static_cast<uint32_t>(h)) << 32) | static_cast<uint32_t>(l));
}
inline float __uint2float_rn(uint32_t x) { return static_cast<float>(x); }
inline float __int2float_rn(int x) { return static_cast<float>(x); }
inline int __float2int_rz(float x) { return static_cast<int>(x); }
inline double __ull2double_rn(uint64_t x) { return static_cast<double>(x); }
inline uint64_t __double2ull_rz(double x) { return x >= 0x1p64 ? ~0ull : static_cast<uint64_t>(x); }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c)
{
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
}
template <typename T> T __ldg(const T *p) { return *p; }
template <typename T, typename F> T atomically(T *p, F f)
{
    T old, next;
    __atomic_load(p, &old, __ATOMIC_RELAXED);
    do next = f(old);
    while (!__atomic_compare_exchange(p, &old, &next, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED));
    return old;
}
template <typename T> T atomicAdd(T *p, T v) { return atomically(p, [v](T x) { return static_cast<T>(x + v); }); }
inline int atomicMin(int *p, int v) { return atomically(p, [v](int x) { return std::min(x, v); }); }
inline int atomicMax(int *p, int v) { return atomically(p, [v](int x) { return std::max(x, v); }); }

// f on every thread of one block.
template <typename F>
void run_block(int threads, F f)
{
    blockDim.x = static_cast<unsigned>(threads);
    for (Meet &m : warps) m.in = m.generation = 0;
    whole_block.in = whole_block.generation = 0;
    std::vector<std::thread> all;
    for (int i = 0; i < threads; ++i)
        all.emplace_back([i, &f] {
            threadIdx.x = static_cast<unsigned>(i);
            f();
        });
    for (std::thread &t : all) t.join();
}
