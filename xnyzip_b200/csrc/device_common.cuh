// Device-side building blocks shared by the XnYZip sm_100a kernels:
//   * warp / block scans, decoupled look-back with bounded waits,
//   * exact float arithmetic of the quantizers (explicit _rn intrinsics, never contracted),
//   * Morton interleave and the table-driven Hilbert transform,
//   * warp-aggregated bit writers and bit readers for the MSB-first (Huffman,
//     exp-Golomb) and LSB-first (Golomb-Rice, bit-packing) streams.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"

namespace xnyz {

using u8 = uint8_t;
using u16 = uint16_t;
using u32 = uint32_t;
using u64 = unsigned long long;  // the type CUDA atomics take
using i32 = int32_t;
using i64 = long long;

constexpr u32 kFullMask = 0xffffffffu;

// Device error bits (OR-ed into a u32 the host reads after each stage).
constexpr u32 kErrTimeout = 1u;      // a bounded wait gave up
constexpr u32 kErrBadStream = 2u;    // a decoder ran past its input or found an invalid code
constexpr u32 kErrOverflow = 4u;     // an output bound was exceeded
constexpr u32 kErrPlacement = 8u;    // a scatter computed a position outside its array (skipped)

// Spin limit for look-back waits: ~1 s with the back-off below, then the waiting thread
// records kErrTimeout and proceeds with what it has (the host reports XNYZ_ERR_TIMEOUT).
constexpr u32 kSpinLimit = 1u << 23;

__device__ __forceinline__ u32 lanemask_lt() {
    u32 m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
__device__ __forceinline__ u32 lane_id() { return threadIdx.x & 31u; }

// ------------------------------------------------------------------ scans ---------------
template <typename T, typename Op>
__device__ __forceinline__ T warp_inclusive(T v, Op op) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        T o = __shfl_up_sync(kFullMask, v, d);
        if ((int)lane_id() >= d) v = op(o, v);
    }
    return v;
}

struct AddOp {
    template <typename T>
    __device__ __forceinline__ T operator()(T a, T b) const { return a + b; }
};

// Warp-wide inclusive sums over the 32 lanes.
template <typename T>
__device__ __forceinline__ T warp_incl_add(T v) {
    const u32 lane = lane_id();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T o = __shfl_up_sync(kFullMask, v, d);
        if (lane >= (u32)d) v += o;
    }
    return v;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFullMask, v, d);
    return v;
}

// Block-wide exclusive scan (THREADS a multiple of 32, <= 1024).  `total` receives the
// block aggregate.  `scratch` holds THREADS/32 + 1 elements of shared memory.
template <int THREADS, typename T, typename Op>
__device__ __forceinline__ T block_exclusive(T v, T identity, Op op, T* scratch, T& total) {
    constexpr int W = THREADS / 32;
    const int w = threadIdx.x >> 5;
    T inc = warp_inclusive(v, op);
    if (lane_id() == 31) scratch[w] = inc;
    __syncthreads();
    if (w == 0) {
        T s = (int)lane_id() < W ? scratch[lane_id()] : identity;
        T si = warp_inclusive(s, op);
        if ((int)lane_id() < W) scratch[lane_id()] = si;  // inclusive over warps
    }
    __syncthreads();
    T warp_prefix = w == 0 ? identity : scratch[w - 1];
    T excl_in_warp = __shfl_up_sync(kFullMask, inc, 1);
    if (lane_id() == 0) excl_in_warp = identity;
    total = scratch[W - 1];
    T r = op(warp_prefix, excl_in_warp);
    __syncthreads();
    return r;
}

// ------------------------------------------------------------- look-back ----------------
__device__ __forceinline__ u32 ld_volatile(const u32* p) { return *(const volatile u32*)p; }
__device__ __forceinline__ u64 ld_volatile(const u64* p) { return *(const volatile u64*)p; }
__device__ __forceinline__ void st_volatile(u32* p, u32 v) { *(volatile u32*)p = v; }
__device__ __forceinline__ void st_volatile(u64* p, u64 v) { *(volatile u64*)p = v; }

// Single-pass chained scans.  A tile publishes its state as one 128-bit word, stored and loaded
// whole, so that neither side needs a fence: lo and the low 62 bits of hi hold the value, the top
// two bits of hi the flag (0 empty, 1 the tile's aggregate, 2 inclusive prefix).  What a value means
// is up to the operator.
using Status = unsigned __int128;
struct Pair {
    u64 lo, hi;
};
__device__ __forceinline__ void st_status(Status* p, Pair v, u32 flag) {
    const Status x = ((Status)(v.hi | ((u64)flag << 62)) << 64) | v.lo;
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(x) : "memory");
}
__device__ __forceinline__ Pair ld_status(const Status* p, u32& flag) {
    Status x;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(x) : "l"(p) : "memory");
    const u64 hi = (u64)(x >> 64);
    flag = (u32)(hi >> 62);
    return Pair{(u64)x, hi & ((1ull << 62) - 1)};
}

// Two sums side by side (lo wraps modulo 2^64, hi stays below 2^62).
struct PairAdd {
    __device__ __forceinline__ Pair operator()(Pair a, Pair b) const { return Pair{a.lo + b.lo, a.hi + b.hi}; }
    // whether nothing before a tile with this value matters to the tiles after it
    __device__ static __forceinline__ bool closed(Pair) { return false; }
};

// Exclusive prefix of `tile` (to every lane), publishing its inclusive prefix; called by all 32 lanes
// of one warp.  Each step reads the states of 128 predecessors, four per lane and the nearest first,
// all in flight together, waits until those up to the nearest inclusive prefix have been published
// and combines them, earlier tiles first (`op` need not commute; {0, 0} is its identity).  A wide
// window matters: with all tiles of a wave publishing at about the same time, the prefixes spread
// by the window per step.  A tile whose value is closed (Op::closed) ends the walk as an inclusive
// prefix does.
template <typename Op>
__device__ Pair chain_lookback(Status* status, u32 tile, Pair mine, Op op, u32* err) {
    const int lane = (int)(threadIdx.x & 31u);
    if (lane == 0) st_status(&status[tile], mine, tile == 0 || Op::closed(mine) ? 2u : 1u);
    if (tile == 0) return Pair{0, 0};
    Pair acc{0, 0};
    i64 top = (i64)tile - 1;
    u32 spins = 0;
    bool failed = false;
    while (true) {
        Pair v[4];
        u32 f[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const i64 q = top - 4 * lane - j;
            f[j] = 2u;
            v[j] = Pair{0, 0};
            if (q >= 0) v[j] = ld_status(&status[q], f[j]);
        }
        Pair r{0, 0};  // my tiles from my nearest inclusive one on
        bool fin = false, empty = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (fin) continue;
            r = op(v[j], r);
            fin = f[j] == 2u;
            empty |= f[j] == 0u;
        }
        const u32 m2 = __ballot_sync(kFullMask, fin);
        const int last = m2 ? __ffs(m2) - 1 : 31;
        if (__any_sync(kFullMask, empty && lane <= last)) {
            if (++spins > kSpinLimit) {
                failed = true;
                break;
            }
            if (spins > 64) __nanosleep(100);
            continue;
        }
        if (lane > last) r = Pair{0, 0};
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const Pair o{__shfl_down_sync(kFullMask, r.lo, d), __shfl_down_sync(kFullMask, r.hi, d)};  // earlier tiles
            if (lane + d < 32) r = op(o, r);
        }
        acc = op(Pair{__shfl_sync(kFullMask, r.lo, 0), __shfl_sync(kFullMask, r.hi, 0)}, acc);
        if (m2) break;
        top -= 128;
    }
    if (lane == 0) {
        if (failed) atomicOr(err, kErrTimeout);
        if (!Op::closed(mine)) st_status(&status[tile], op(acc, mine), 2u);
    }
    return acc;
}

__device__ __forceinline__ u64 chain_add(void* status, u32 tile, u64 mine, u32* err) {
    return chain_lookback(static_cast<Status*>(status), tile, Pair{mine, 0}, PairAdd{}, err).lo;
}

// Dynamic tile index: tiles are claimed in launch order, so a tile's predecessors have
// all started before it waits on them.
__device__ __forceinline__ u32 claim_tile(u32* counter, u32* smem_slot) {
    if (threadIdx.x == 0) *smem_slot = atomicAdd(counter, 1u);
    __syncthreads();
    return *smem_slot;
}

// ------------------------------------------------------------ quantizers ----------------
// Quantizer constants (dev::QuantParams) are derived on the host exactly as the reference
// derives them: div = float(double(2.0f * l2) / sqrt(5 or 3)) (quantize divisor), s = l2,
// rdiv = float(sqrt(5 or 3)) (recover: ((v * 2) * s) / rdiv).
using dev::QuantParams;

// x / d correctly rounded, given y = RN(1 / d): one fused correction of x y (P. Markstein, IBM J. Res.
// Dev. 34(1), 1990).  Used for the two constants sqrt(3) and sqrt(5) rounded to float, for which every
// significand has been compared with IEEE division, and for |x| far from underflow and overflow.
__device__ __forceinline__ float div_const(float x, float d, float y) {
    const float q = __fmul_rn(x, y);
    return __fmaf_rn(__fmaf_rn(-q, d, x), y, q);
}

// x / d correctly rounded for any divisor whose significand is not all ones, given y = RN(1 / d): two
// corrections, the first of which makes the quotient faithful (P. Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, 1990).  x is 0 or in [2^-60, 2^60], d in [2^-42, 2^42]: the remainders are exact.
__device__ __forceinline__ float div_any(float x, float d, float y) {
    float q = __fmul_rn(x, y);
    q = __fmaf_rn(__fmaf_rn(-q, d, x), y, q);
    return __fmaf_rn(__fmaf_rn(-q, d, x), y, q);
}

// static_cast<int>(float) as compiled for x86-64 (cvttss2si): truncation toward zero and
// 0x80000000 for NaN or values outside the int range.
__device__ __forceinline__ i32 f2i_x86(float f) {
    if (!(f > -2147483904.0f && f < 2147483648.0f)) return (i32)0x80000000;
    return __float2int_rz(f);
}

__device__ __forceinline__ float sqf(float a) { return __fmul_rn(a, a); }

// Truncated-octahedron (BCC) quantizer: nearest of the even and odd cubic lattices with
// the reference's coefficient-wise float operations, then x,y halved (quantizer/
// truncated_octahedron_quantizer.hpp:21-55).  squaredNorm sums as c0 + (c1 + c2).
__device__ __forceinline__ void quantize_to(float px, float py, float pz, float div, i32& ox, i32& oy, i32& oz) {
    const float q0 = __fdiv_rn(px, div), q1 = __fdiv_rn(py, div), q2 = __fdiv_rn(pz, div);
    const float e0 = __fmul_rn(roundf(__fmul_rn(q0, 0.5f)), 2.0f);
    const float e1 = __fmul_rn(roundf(__fmul_rn(q1, 0.5f)), 2.0f);
    const float e2 = __fmul_rn(roundf(__fmul_rn(q2, 0.5f)), 2.0f);
    const float o0 = __fadd_rn(__fmul_rn(roundf(__fmul_rn(__fsub_rn(q0, 1.0f), 0.5f)), 2.0f), 1.0f);
    const float o1 = __fadd_rn(__fmul_rn(roundf(__fmul_rn(__fsub_rn(q1, 1.0f), 0.5f)), 2.0f), 1.0f);
    const float o2 = __fadd_rn(__fmul_rn(roundf(__fmul_rn(__fsub_rn(q2, 1.0f), 0.5f)), 2.0f), 1.0f);
    const float dE = __fadd_rn(sqf(__fsub_rn(q0, e0)), __fadd_rn(sqf(__fsub_rn(q1, e1)), sqf(__fsub_rn(q2, e2))));
    const float dO = __fadd_rn(sqf(__fsub_rn(q0, o0)), __fadd_rn(sqf(__fsub_rn(q1, o1)), sqf(__fsub_rn(q2, o2))));
    i32 n0, n1, n2;
    if (dE <= dO) {
        n0 = f2i_x86(e0); n1 = f2i_x86(e1); n2 = f2i_x86(e2);
    } else {
        n0 = f2i_x86(o0); n1 = f2i_x86(o1); n2 = f2i_x86(o2);
    }
    if (n0 & 1) {
        n0 = (i32)((u32)n0 + 1u) >> 1;
        n1 = (i32)((u32)n1 + 1u) >> 1;
    } else {
        n0 >>= 1;
        n1 >>= 1;
    }
    ox = n0; oy = n1; oz = n2;
}

// Cube quantizer: floor(p / div) (quantizer/cube_quantizer.hpp:15-27).
__device__ __forceinline__ void quantize_cube(float px, float py, float pz, float div, i32& ox, i32& oy, i32& oz) {
    ox = f2i_x86(floorf(__fdiv_rn(px, div)));
    oy = f2i_x86(floorf(__fdiv_rn(py, div)));
    oz = f2i_x86(floorf(__fdiv_rn(pz, div)));
}

// Adaptive quantizer steps: from device memory while compressing, from the container's
// parameters while decompressing.
__device__ __forceinline__ float adaptive_step(const QuantParams& q, int a) {
    return q.step_dev ? q.step_dev[a] : q.step[a];
}

// Adaptive quantizer: round(p / step) per axis, half away from zero, then the x86 cast
// (quantizer/adaptive_quantizer.hpp:66-77).
__device__ __forceinline__ void quantize_adaptive(const QuantParams& q, float px, float py, float pz, i32& ox,
                                                  i32& oy, i32& oz) {
    ox = f2i_x86(roundf(__fdiv_rn(px, adaptive_step(q, 0))));
    oy = f2i_x86(roundf(__fdiv_rn(py, adaptive_step(q, 1))));
    oz = f2i_x86(roundf(__fdiv_rn(pz, adaptive_step(q, 2))));
}

__device__ __forceinline__ void quantize(const QuantParams& q, float px, float py, float pz, i32& ox, i32& oy,
                                         i32& oz) {
    if (q.quantizer == 1)
        quantize_to(px, py, pz, q.div, ox, oy, oz);
    else if (q.quantizer == 2)
        quantize_adaptive(q, px, py, pz, ox, oy, oz);
    else
        quantize_cube(px, py, pz, q.div, ox, oy, oz);
}

// Recover + unshift (truncated_octahedron_quantizer.hpp:57-76, cube_quantizer.hpp:29-38,
// adaptive_quantizer.hpp:83-97: idx * step, shifting.hpp:39-50).
__device__ __forceinline__ void recover(const QuantParams& q, i32 cx, i32 cy, i32 cz, float offx, float offy,
                                        float offz, float& x, float& y, float& z) {
    float fx, fy, fz;
    if (q.quantizer == 1) {
        i32 nx, ny;
        if (cz & 1) {
            nx = (i32)(((u32)cx << 1) - 1u);
            ny = (i32)(((u32)cy << 1) - 1u);
        } else {
            nx = (i32)((u32)cx << 1);
            ny = (i32)((u32)cy << 1);
        }
        fx = __fdiv_rn(__fmul_rn(__fmul_rn(__int2float_rn(nx), 2.0f), q.s), q.rdiv);
        fy = __fdiv_rn(__fmul_rn(__fmul_rn(__int2float_rn(ny), 2.0f), q.s), q.rdiv);
        fz = __fdiv_rn(__fmul_rn(__fmul_rn(__int2float_rn(cz), 2.0f), q.s), q.rdiv);
    } else if (q.quantizer == 2) {
        fx = __fmul_rn(__int2float_rn(cx), adaptive_step(q, 0));
        fy = __fmul_rn(__int2float_rn(cy), adaptive_step(q, 1));
        fz = __fmul_rn(__int2float_rn(cz), adaptive_step(q, 2));
    } else {
        fx = __fdiv_rn(__fmul_rn(__fmul_rn(__fadd_rn(__int2float_rn(cx), 0.5f), 2.0f), q.s), q.rdiv);
        fy = __fdiv_rn(__fmul_rn(__fmul_rn(__fadd_rn(__int2float_rn(cy), 0.5f), 2.0f), q.s), q.rdiv);
        fz = __fdiv_rn(__fmul_rn(__fmul_rn(__fadd_rn(__int2float_rn(cz), 0.5f), 2.0f), q.s), q.rdiv);
    }
    x = __fadd_rn(fx, offx);
    y = __fadd_rn(fy, offy);
    z = __fadd_rn(fz, offz);
}

// ------------------------------------------------------------------ Morton ---------------
// 21 bits per axis interleaved x (bit 0), y (bit 1), z (bit 2) (preprocessor/
// z_order_curve.hpp:14-47), with the usual mask cascade.
__device__ __forceinline__ u64 spread3(u32 v) {
    u64 x = v & 0x1fffffu;
    x = (x | (x << 32)) & 0x001f00000000ffffull;
    x = (x | (x << 16)) & 0x001f0000ff0000ffull;
    x = (x | (x << 8)) & 0x100f00f00f00f00full;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}
__device__ __forceinline__ u32 gather3(u64 m) {
    u64 x = m & 0x1249249249249249ull;
    x = (x | (x >> 2)) & 0x10c30c30c30c30c3ull;
    x = (x | (x >> 4)) & 0x100f00f00f00f00full;
    x = (x | (x >> 8)) & 0x001f0000ff0000ffull;
    x = (x | (x >> 16)) & 0x001f00000000ffffull;
    x = (x | (x >> 32)) & 0x1fffffull;
    return (u32)x;
}
__device__ __forceinline__ u64 morton3(i32 x, i32 y, i32 z) {
    return spread3((u32)x) | (spread3((u32)y) << 1) | (spread3((u32)z) << 2);
}

// ------------------------------------------------------------------ Hilbert --------------
// Table-driven digit transform.  A state is one orientation of the curve (an element of
// the cube's rotation group, <= 32 states); entry [state*8 + digit] holds the output digit
// in bits 0-2 and the next state in bits 3-7.  Levels above `top` are left unchanged, as
// in mortonToHilbert3 / hilbertToMorton3 with iteration = top.
__device__ __forceinline__ u64 hilbert_apply(const u8* tab, u64 code, int top, u32 state) {
    u64 out = top >= 20 ? (code & (top >= 21 ? 0ull : ~0ull << 63)) : (code & (~0ull << (3 * (top + 1))));
    for (int l = top; l >= 0; --l) {
        const u32 d = (u32)(code >> (3 * l)) & 7u;
        const u32 e = tab[state * 8 + d];
        out |= (u64)(e & 7u) << (3 * l);
        state = e >> 3;
    }
    return out;
}

// gather3 of hilbert_apply(tab, code, top, state) for each axis: the output digit of level
// l is bit l of x, y and z (bits 0, 1, 2 of the digit), so the transformed levels are
// de-interleaved as they are produced; levels above `top` pass through gather3.
__device__ __forceinline__ void hilbert_xyz(const u8* tab, u64 code, int top, u32 state, u32& x, u32& y, u32& z) {
    const u64 above = top >= 20 ? (code & (top >= 21 ? 0ull : ~0ull << 63)) : (code & (~0ull << (3 * (top + 1))));
    x = y = z = 0;
    if (above) {
        x = gather3(above);
        y = gather3(above >> 1);
        z = gather3(above >> 2);
    }
    for (int l = top; l >= 0; --l) {
        const u32 e = tab[state * 8 + ((u32)(code >> (3 * l)) & 7u)];
        x |= (e & 1u) << l;
        y |= ((e >> 1) & 1u) << l;
        z |= ((e >> 2) & 1u) << l;
        state = e >> 3;
    }
}

// ------------------------------------------------------------- bit writers --------------
// Stream words are 32-bit; the output buffer must be zeroed and 4-byte aligned.
// MSB-first streams: stream bit p is bit (7 - p%8) of byte p/8; a 32-bit word k then holds
// stream bits [32k, 32k+32) most significant first, stored byte-swapped in memory.
// LSB-first streams: stream bit p is bit p%8 of byte p/8 = bit p%32 of little-endian word k.
//
// Every lane of a warp calls these together (inactive lanes pass nbits = 0).  Lanes must
// pass non-decreasing positions in lane order (true for scan-derived offsets); the writes
// of lanes landing in the same word are OR-combined with shuffles first, so one atomicOr
// per distinct word and warp reaches memory.
__device__ __forceinline__ void warp_or_word(u32* words, u64 word, u32 bits, bool active) {
    // Segmented OR over lanes with equal `word` (non-decreasing across lanes).
    const u32 lane = lane_id();
    const int act = active ? 1 : 0;
    u32 v = active ? bits : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        u32 ov = __shfl_up_sync(kFullMask, v, d);
        u64 ow = __shfl_up_sync(kFullMask, word, d);
        int oa = __shfl_up_sync(kFullMask, act, d);
        if ((int)lane >= d && oa && ow == word) v |= ov;
    }
    u64 nw = __shfl_down_sync(kFullMask, word, 1);
    int na = __shfl_down_sync(kFullMask, act, 1);
    bool last = (lane == 31) || !na || nw != word;
    if (active && last && v) atomicOr(&words[word], v);
}

// One thread's run of consecutive codes of an MSB-first stream, from stream bit `pos` on
// (begin / put / end).  Bits collect in a 64-bit buffer and leave a word at a time: the
// run's first and last words may be shared with the neighbouring runs and are OR-ed in
// atomically, the words in between belong to this run alone and are stored.  For short codes
// this is one or two memory operations per run instead of one per code.
struct MsbRun {
    u32* words;
    u64 k;    // word that buf's first bit belongs to
    u64 buf;  // pending bits, first in bit 63
    u32 nb;   // pending bits (< 32 between puts)
    bool first;
    __device__ __forceinline__ void begin(u32* w, u64 pos) {
        words = w;
        k = pos >> 5;
        nb = (u32)(pos & 31u);  // the word's leading bits belong to the previous run: zeros here
        buf = 0;
        first = true;
    }
    __device__ __forceinline__ void flush() {
        const u32 wv = __byte_perm((u32)(buf >> 32), 0, 0x0123);
        if (first) {
            if (wv) atomicOr(&words[k], wv);
            first = false;
        } else {
            words[k] = wv;
        }
        buf <<= 32;
        nb -= 32;
        ++k;
    }
    // the low n (<= 32) bits of v, most significant first
    __device__ __forceinline__ void put32(u32 v, u32 n) {
        if (!n) return;
        if (nb >= 32) flush();
        buf |= ((u64)v << (64u - n)) >> nb;
        nb += n;
    }
    __device__ __forceinline__ void zeros(u64 n) {
        while (n) {
            const u32 t = n > 32 ? 32u : (u32)n;
            put32(0u, t);
            n -= t;
        }
    }
    // the low n (<= 64) bits of v, most significant first
    __device__ __forceinline__ void put(u64 v, u32 n) {
        if (n > 32) {
            put32((u32)(v >> 32), n - 32);
            put32((u32)v, 32);
        } else {
            put32((u32)v, n);
        }
    }
    __device__ __forceinline__ void end() {
        if (nb >= 32) flush();
        if (nb) {  // the last word, shared with the next run
            const u32 wv = __byte_perm((u32)(buf >> 32), 0, 0x0123);
            if (wv) atomicOr(&words[k], wv);
        }
    }
};

// The LSB-first counterpart of MsbRun: bits collect from bit 0 of the buffer up.
struct LsbRun {
    u32* words;
    u64 k;
    u64 buf;  // pending bits, first in bit 0
    u32 nb;
    bool first;
    __device__ __forceinline__ void begin(u32* w, u64 pos) {
        words = w;
        k = pos >> 5;
        nb = (u32)(pos & 31u);
        buf = 0;
        first = true;
    }
    __device__ __forceinline__ void flush() {
        const u32 wv = (u32)buf;
        if (first) {
            if (wv) atomicOr(&words[k], wv);
            first = false;
        } else {
            words[k] = wv;
        }
        buf >>= 32;
        nb -= 32;
        ++k;
    }
    // the low n (<= 32) bits of v, least significant first
    __device__ __forceinline__ void put32(u32 v, u32 n) {
        if (!n) return;
        if (nb >= 32) flush();
        buf |= (u64)(n == 32u ? v : (v & ((1u << n) - 1u))) << nb;
        nb += n;
    }
    __device__ __forceinline__ void ones(u64 n) {
        while (n) {
            const u32 t = n > 32 ? 32u : (u32)n;
            put32(0xffffffffu, t);
            n -= t;
        }
    }
    __device__ __forceinline__ void put(u64 v, u32 n) {
        if (n > 32) {
            put32((u32)v, 32);
            put32((u32)(v >> 32), n - 32);
        } else {
            put32((u32)v, n);
        }
    }
    __device__ __forceinline__ void end() {
        if (nb >= 32) flush();
        if (nb) {
            const u32 wv = (u32)buf;
            if (wv) atomicOr(&words[k], wv);
        }
    }
};

// Writes `nbits` (<= 64) bits of `val`, least significant first, at position `pos` of an
// LSB-first stream.
__device__ __forceinline__ void warp_write_lsb(u32* words, u64 pos, u64 val, u32 nbits) {
    const bool act = nbits != 0;
    const u64 k0 = pos >> 5;
    const u32 o = (u32)(pos & 31u);
    unsigned __int128 chunk = 0;
    if (act) {
        const u64 v = nbits == 64 ? val : (val & ((1ull << nbits) - 1));
        chunk = (unsigned __int128)v << o;
    }
    const u32 w0 = (u32)chunk, w1 = (u32)(chunk >> 32), w2 = (u32)(chunk >> 64);
    warp_or_word(words, k0, w0, act);
    if (__any_sync(kFullMask, act && w1 != 0u)) warp_or_word(words, k0 + 1, w1, act);
    if (__any_sync(kFullMask, act && w2 != 0u)) warp_or_word(words, k0 + 2, w2, act);
}

__device__ __forceinline__ u32 bitlen64(u64 v) { return v ? 64u - (u32)__clzll((long long)v) : 0u; }

}  // namespace xnyz
