// Point-level kernels: bounding-box minimum (shift_points), quantization with range and
// error statistics, and sort-key generation for block and direct mode.
//
// Reference behaviour restated here (paths relative to the reference's source/):
//   shift_points           preprocessor/shifting.hpp:11-36  (strict '<' scan from FLT_MAX)
//   quantize               quantizer/truncated_octahedron_quantizer.hpp:21-55, cube_quantizer.hpp:15-27,
//                          adaptive_quantizer.hpp:16-81
//   ranges / direct switch composer/block_compressor.hpp:69-88
//   error statistics       composer/block_compressor_rle.hpp:53-67
//   block keys             quantizer/block_quantizer.hpp:93-115
//   direct keys            composer/block_compressor.hpp:90-101
#include <cfloat>

#include "device_common.cuh"
#include "kernels.h"

namespace xnyz {
namespace dev {

namespace {

constexpr int kThreads = 256;

// Grid-stride loop over points that issues the loads of U points (U strides apart) before
// processing them, so that each thread keeps U loads in flight.  body(i, x, y, z).
template <int U, typename F>
__device__ __forceinline__ void for_each_point(const float* __restrict__ xyz, u64 n, F&& body) {
    const u64 stride = (u64)gridDim.x * kThreads;
    for (u64 i0 = (u64)blockIdx.x * kThreads + threadIdx.x; i0 < n; i0 += U * stride) {
        float x[U], y[U], z[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const u64 i = i0 + (u64)u * stride;
            if (i < n) {
                x[u] = __ldg(xyz + 3 * i);
                y[u] = __ldg(xyz + 3 * i + 1);
                z[u] = __ldg(xyz + 3 * i + 2);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const u64 i = i0 + (u64)u * stride;
            if (i < n) body(i, x[u], y[u], z[u]);
        }
    }
}

// At kVecPoints points and more, and with 16-byte aligned arrays, a thread takes four neighbouring
// points at a time, as three 16-byte loads; below, one at a time, so that small inputs fill the chip
// (at 1M points quantization takes 16.7 us so and 18.0 one by one, at 120k they are equal).
constexpr u64 kVecPoints = 1ull << 18;
inline bool use_vec(u64 n, const void* a, const void* b = nullptr) {
    return n >= kVecPoints && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}

// Order key of a float for the minimum scan: monotone in value, +0 and -0 equal, NaN last.
__device__ __forceinline__ u32 order_key(float f) {
    u32 b = __float_as_uint(f);
    if ((b & 0x7fffffffu) > 0x7f800000u) return 0xffffffffu;  // NaN never wins ('<' is false)
    if ((b & 0x7fffffffu) == 0u) b = 0u;                        // -0 ties with +0
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ unsigned long long umin64(unsigned long long a, unsigned long long b) { return a < b ? a : b; }

// Minimum over the block of three u64 values, then one atomicMin per axis.
__device__ void block_min3(unsigned long long m[3], unsigned long long* dst) {
    __shared__ unsigned long long sm[3][kThreads / 32];
    for (int a = 0; a < 3; ++a) {
        unsigned long long v = m[a];
        for (int d = 16; d > 0; d >>= 1) v = umin64(v, __shfl_xor_sync(kFullMask, v, d));
        if (lane_id() == 0) sm[a][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        unsigned long long v = sm[threadIdx.x][0];
        for (int w = 1; w < kThreads / 32; ++w) v = umin64(v, sm[threadIdx.x][w]);
        atomicMin(&dst[threadIdx.x], v);
    }
}

// Maximum over the block of three u32 order keys, then one atomicMax per axis.
__device__ void block_max3(u32 m[3], unsigned int* dst) {
    __shared__ u32 sm[3][kThreads / 32];
    for (int a = 0; a < 3; ++a) {
        u32 v = m[a];
        for (int d = 16; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(kFullMask, v, d));
        if (lane_id() == 0) sm[a][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        u32 v = sm[threadIdx.x][0];
        for (int w = 1; w < kThreads / 32; ++w) v = max(v, sm[threadIdx.x][w]);
        atomicMax(&dst[threadIdx.x], v);
    }
}

// shift_points keeps the first of equal minima; the key packs (order key, index) so the
// smallest index wins ties (including +0 / -0), and the initial FLT_MAX candidate carries
// index 0xffffffff.  The largest order key per axis feeds the adaptive quantizer's steps.
__global__ void __launch_bounds__(kThreads) bbox_kernel(const float* __restrict__ xyz, u64 n, PointStats* stats) {
    unsigned long long m[3];
    u32 mx[3];
    for (int a = 0; a < 3; ++a) {
        m[a] = ~0ull;
        mx[a] = 0u;
    }
    for_each_point<4>(xyz, n, [&](u64 i, float x, float y, float z) {
        const float v[3] = {x, y, z};
        for (int a = 0; a < 3; ++a) {
            const u32 ok = order_key(v[a]);
            m[a] = umin64(m[a], ((unsigned long long)ok << 32) | (u32)i);
            mx[a] = max(mx[a], ok);
        }
    });
    block_min3(m, stats->minkey);
    block_max3(mx, stats->maxkey);
}

// The same in 16-byte pieces.  Piece k holds floats [4 k, 4 k + 4), of axes (k + j) % 3; the grid's
// threads are a multiple of three, so that a thread's pieces all start on the same axis p = k % 3 and it
// keeps three minima, relative to p, by the scan's own '<' (a key per point cost 68 instructions, and
// 183 us for 64M points; this 144, 5.3 TB/s).
__global__ void __launch_bounds__(kThreads) bbox_vec_kernel(const float* __restrict__ xyz, u64 n, PointStats* stats) {
    const u64 pieces = 3 * n / 4, stride = (u64)gridDim.x * kThreads;
    const u64 k0 = (u64)blockIdx.x * kThreads + threadIdx.x;
    const u32 p = (u32)(k0 % 3u);
    const float4* v4 = reinterpret_cast<const float4*>(xyz);
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    u32 at[3] = {~0u, ~0u, ~0u};
    u32 first = (u32)(k0 / 3u) * 4u;             // the piece's points, less (4 p + j) / 3
    const u32 step = (u32)(stride / 3u) * 4u;
    const u32 o[4] = {4u * p / 3u, (4u * p + 1u) / 3u, (4u * p + 2u) / 3u, (4u * p + 3u) / 3u};
    auto take = [&](int j, float x, u32 i) {
        if (x < lo[j]) {
            lo[j] = x;
            at[j] = i;
        }
        hi[j] = fmaxf(hi[j], x);
    };
    for (u64 k = k0; k < pieces; k += 4 * stride) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k + u * stride < pieces) v[u] = __ldg(v4 + k + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (k + u * stride < pieces) {
                take(0, v[u].x, first + o[0]);
                take(1, v[u].y, first + o[1]);
                take(2, v[u].z, first + o[2]);
                take(0, v[u].w, first + o[3]);
            }
            first += step;
        }
    }
    unsigned long long m[3];
    u32 mx[3];
#pragma unroll
    for (u32 a = 0; a < 3; ++a) {
        const u32 j = a >= p ? a - p : a + 3u - p;
        const float l = j == 0 ? lo[0] : j == 1 ? lo[1] : lo[2];
        const float h = j == 0 ? hi[0] : j == 1 ? hi[1] : hi[2];
        const u32 i = j == 0 ? at[0] : j == 1 ? at[1] : at[2];
        m[a] = ((unsigned long long)order_key(l) << 32) | i;
        mx[a] = order_key(h);
    }
    const u64 rest = 4 * pieces + k0;  // the floats after the last piece, one each
    if (rest < 3 * n) {
        const u32 ok = order_key(xyz[rest]), a = (u32)(rest % 3u);
        m[a] = umin64(m[a], ((unsigned long long)ok << 32) | (u32)(rest / 3u));
        mx[a] = max(mx[a], ok);
    }
    block_min3(m, stats->minkey);
    block_max3(mx, stats->maxkey);
}

__device__ __forceinline__ float order_key_value(u32 k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ void load_offset(const float* xyz, const PointStats* st, float off[3]) {
    for (int a = 0; a < 3; ++a) {
        const unsigned long long k = st->minkey[a];
        const u32 idx = (u32)(k & 0xffffffffu);
        const u32 ok = (u32)(k >> 32);
        // The reference starts from FLT_MAX; a candidate wins only if strictly smaller.
        off[a] = (idx == 0xffffffffu || ok >= order_key(FLT_MAX)) ? FLT_MAX : xyz[3 * (u64)idx + a];
    }
}

__device__ __forceinline__ bool finite3(float x, float y, float z) {
    return isfinite(x) && isfinite(y) && isfinite(z);
}

// AdaptiveQuantizer::quantize's steps (quantizer/adaptive_quantizer.hpp:42-64).  Over the
// shifted points the minimum is 0 (the offset is the minimum) and the maximum is
// max - offset (float subtraction is monotone), each compared against the scan's start
// values (FLT_MAX, and the smallest normal float for the maxima).  One thread, IEEE
// single-precision operations in the reference's order.
__global__ void adaptive_steps_kernel(const float* __restrict__ xyz, float R, PointStats* stats) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    float off[3];
    load_offset(xyz, stats, off);
    float d[3];
    for (int a = 0; a < 3; ++a) {
        const float hi = __fsub_rn(order_key_value(stats->maxkey[a]), off[a]);
        const float mx = (FLT_MIN < hi) ? hi : FLT_MIN;
        const float lo = __fsub_rn(off[a], off[a]);  // the minimum's own shifted value
        const float mn = (lo < FLT_MAX) ? lo : FLT_MAX;
        d[a] = __fsub_rn(mx, mn);
    }
    const float norm = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])),
                                            __fmul_rn(d[2], d[2])));
    for (int a = 0; a < 3; ++a)
        stats->step[a] = norm > 0.0f ? __fdiv_rn(__fmul_rn(R, d[a]), norm) : __fdiv_rn(R, __fsqrt_rn(3.0f));
}

// quantize and recover (offset 0) of a point whose coordinates are 0 or at least 2^-60 and whose
// quotients are below 2^24, in a third of the instructions: the divisions by multiplication, the lattice
// neighbours from the quotient's floor, the recovered coordinates from the lattice values as floats.
//
// The truncated octahedron's candidates are round(q / 2) * 2 and round((q - 1) / 2) * 2 + 1, half away
// from zero, in single precision.  For q >= 0 that is, by the parity of f = floor(q): f or f + 1.  The
// halves are exact, and so is q - 1 but for q < 1/2, where it matters only at q <= 2^-25: it rounds to
// -1 there, and the odd candidate is -1.
template <int QUANT>
__device__ __forceinline__ void quantize_small(const QuantParams& q, const float (&p)[3], i32 (&c)[3], float (&r)[3]) {
    float t[3], v[3];
    i32 f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        t[a] = div_any(p[a], q.div, q.inv);
        f[a] = __float2int_rd(t[a]);
    }
    if (QUANT == 1) {
        float e[3], o[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float fl = __int2float_rn(f[a]), up = __fadd_rn(fl, 1.0f);
            const bool odd = f[a] & 1;
            e[a] = odd ? up : fl;
            o[a] = t[a] <= 0x1p-25f ? -1.0f : odd ? fl : up;
        }
        const float dE = __fadd_rn(sqf(__fsub_rn(t[0], e[0])), __fadd_rn(sqf(__fsub_rn(t[1], e[1])), sqf(__fsub_rn(t[2], e[2]))));
        const float dO = __fadd_rn(sqf(__fsub_rn(t[0], o[0])), __fadd_rn(sqf(__fsub_rn(t[1], o[1])), sqf(__fsub_rn(t[2], o[2]))));
        const bool even = dE <= dO;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            v[a] = even ? e[a] : o[a];
            // the lattice value: even f or f + 1, odd f or f + 1 or -1; x and y are halved, upwards
            const i32 n = even ? f[a] + (f[a] & 1) : t[a] <= 0x1p-25f ? -1 : f[a] | 1;
            c[a] = a < 2 ? (n + 1) >> 1 : n;
        }
    } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            c[a] = f[a];
            v[a] = __fadd_rn(__int2float_rn(f[a]), 0.5f);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) r[a] = __fadd_rn(div_const(__fmul_rn(v[a], 2.0f * q.s), q.rdiv, q.rinv), 0.0f);
}

// The cells of all points, their range and the error statistics.  Bound by instructions: with divisions,
// rounding functions and 4-byte accesses it took 232 per point and 536 us for 64M points; this 353, 4.4 TB/s.
template <bool VEC>
__global__ void __launch_bounds__(kThreads) quantize_range_kernel(const float* __restrict__ xyz, u64 n,
                                                                  QuantParams q, PointStats* stats,
                                                                  int with_error_stats, i32* __restrict__ cells) {
    __shared__ float off[3];
    __shared__ int small;
    __shared__ int smax[3][kThreads / 32], smin[3][kThreads / 32];
    __shared__ u32 snf[kThreads / 32], smse[kThreads / 32];
    __shared__ double ssum[kThreads / 32];
    if (threadIdx.x == 0) {
        load_offset(xyz, stats, off);
        bool ok = q.quantizer != 2 && q.inv != 0.0f;
        for (int a = 0; a < 3; ++a) {
            const float extent = __fsub_rn(order_key_value(stats->maxkey[a]), off[a]);
            ok &= extent < 0x1p60f && extent * q.inv < 16000000.0f;  // (a NaN is not)
        }
        small = ok;
        if (blockIdx.x == 0)
            for (int a = 0; a < 3; ++a) stats->offset[a] = off[a];
    }
    __syncthreads();
    const float ox = off[0], oy = off[1], oz = off[2];
    const bool fast = small;
    int mx[3] = {0, 0, 0};
    int mn[3] = {INT_MAX, INT_MAX, INT_MAX};
    u32 nonfinite = 0;
    float emax = 0.0f;
    double esum = 0.0;
    // the point's cell; a point that is not finite has none, is counted and keeps what c holds
    auto point = [&](float x, float y, float z, i32 (&c)[3]) {
        if (!finite3(x, y, z)) {
            ++nonfinite;
            return false;
        }
        const float p[3] = {__fsub_rn(x, ox), __fsub_rn(y, oy), __fsub_rn(z, oz)};
        float r[3];
        // (0 - 1 is the largest)
        const u32 least = min(min(__float_as_uint(p[0]) - 1u, __float_as_uint(p[1]) - 1u), __float_as_uint(p[2]) - 1u);
        if (fast && least >= 0x21800000u - 1u) {  // 2^-60
            if (q.quantizer == 1) quantize_small<1>(q, p, c, r);
            else quantize_small<0>(q, p, c, r);
        } else {
            quantize(q, p[0], p[1], p[2], c[0], c[1], c[2]);
            recover(q, c[0], c[1], c[2], 0.0f, 0.0f, 0.0f, r[0], r[1], r[2]);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            mx[a] = max(mx[a], c[a]);
            mn[a] = min(mn[a], c[a]);
        }
        if (with_error_stats) {
            // (sx - rx)^2 + (sy - ry)^2 + (sz - rz)^2 in float, left to right.
            const float e = __fadd_rn(__fadd_rn(sqf(__fsub_rn(p[0], r[0])), sqf(__fsub_rn(p[1], r[1]))), sqf(__fsub_rn(p[2], r[2])));
            emax = fmaxf(emax, e);
            esum += (double)e;
        }
        return true;
    };
    auto one = [&](u64 i, float x, float y, float z) {
        i32 c[3];
        if (point(x, y, z, c) && cells) {  // kept for the key kernel (keys_cells_kernel), which then need not quantize again
            cells[3 * i] = c[0];
            cells[3 * i + 1] = c[1];
            cells[3 * i + 2] = c[2];
        }
    };
    if (VEC) {
        const u64 quads = n / 4, stride = (u64)gridDim.x * kThreads, k0 = (u64)blockIdx.x * kThreads + threadIdx.x;
        for (u64 k = k0; k < quads; k += stride) {
            const float4* src = reinterpret_cast<const float4*>(xyz) + 3 * k;
            const float4 v0 = __ldg(src), v1 = __ldg(src + 1), v2 = __ldg(src + 2);
            i32 c[4][3] = {};
            point(v0.x, v0.y, v0.z, c[0]);
            point(v0.w, v1.x, v1.y, c[1]);
            point(v1.z, v1.w, v2.x, c[2]);
            point(v2.y, v2.z, v2.w, c[3]);
            if (cells) {
                int4* dst = reinterpret_cast<int4*>(cells) + 3 * k;
                dst[0] = make_int4(c[0][0], c[0][1], c[0][2], c[1][0]);
                dst[1] = make_int4(c[1][1], c[1][2], c[2][0], c[2][1]);
                dst[2] = make_int4(c[2][2], c[3][0], c[3][1], c[3][2]);
            }
        }
        const u64 i = 4 * quads + k0;
        if (i < n) one(i, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
    } else {
        for_each_point<4>(xyz, n, one);
    }
    for (int d = 16; d > 0; d >>= 1) {
        for (int a = 0; a < 3; ++a) {
            mx[a] = max(mx[a], __shfl_xor_sync(kFullMask, mx[a], d));
            mn[a] = min(mn[a], __shfl_xor_sync(kFullMask, mn[a], d));
        }
        nonfinite += __shfl_xor_sync(kFullMask, nonfinite, d);
        emax = fmaxf(emax, __shfl_xor_sync(kFullMask, emax, d));
        esum += __shfl_xor_sync(kFullMask, esum, d);
    }
    const int w = threadIdx.x >> 5;
    if (lane_id() == 0) {
        for (int a = 0; a < 3; ++a) {
            smax[a][w] = mx[a];
            smin[a][w] = mn[a];
        }
        snf[w] = nonfinite;
        smse[w] = __float_as_uint(emax);
        ssum[w] = esum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int bx[3] = {0, 0, 0}, bn[3] = {INT_MAX, INT_MAX, INT_MAX};
        u32 nf = 0, em = 0;
        double es = 0.0;
        for (int k = 0; k < kThreads / 32; ++k) {
            for (int a = 0; a < 3; ++a) {
                bx[a] = max(bx[a], smax[a][k]);
                bn[a] = min(bn[a], smin[a][k]);
            }
            nf += snf[k];
            em = max(em, smse[k]);
            es += ssum[k];
        }
        for (int a = 0; a < 3; ++a) {
            atomicMax(&stats->max_cell[a], bx[a]);
            atomicMin(&stats->min_cell[a], bn[a]);
        }
        if (nf) atomicAdd(&stats->nonfinite, nf);
        if (with_error_stats) {
            atomicMax(&stats->mse_max_bits, em);
            atomicAdd(&stats->mse_sum, es);
        }
    }
}

// Per-block histograms of the sort digits, flushed with one atomicAdd per non-zero bin.
struct DigitHist {
    u32* s;  // shared [passes * 256]
    int passes;
    __device__ __forceinline__ void add(u64 key) {
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (p < passes) atomicAdd(&s[p * 256 + (u32)((key >> (8 * p)) & 255u)], 1u);
    }
};

__device__ __forceinline__ void stage_hilbert_table(const u8* g, u8* s) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s[i] = g ? g[i] : 0;
}

// Block mode: key = id << 21 | quad << 18 | sfc18 of a cell with x, y >= 0 and z >= -1 (checked before);
// z = -1 wraps to 2^64 - 1 before the reference's division by 64 (size_t arithmetic).  Two Hilbert levels
// per read of the table.
__device__ __forceinline__ u64 block_key(i32 x, i32 y, i32 z, const BlockKeyParams& kp, const unsigned short* tab2) {
    const u32 X = (u32)x, Y = (u32)y, Z = (u32)z;
    u32 low = ((X >> 6) & 1u) | (((Y >> 6) & 1u) << 1) | (((Z >> 6) & 1u) << 2);
    if (kp.hilbert) {
        u32 s = kp.hstart << 6;
#pragma unroll
        for (int l = 2; l >= 0; --l) {
            const u32 d = ((X >> (2 * l)) & 3u) | (((Y >> (2 * l)) & 3u) << 2) | (((Z >> (2 * l)) & 3u) << 4);
            s = tab2[(s & ~63u) | d];
            low = (low << 6) | (s & 63u);
        }
    } else {
        auto spread = [](u32 v) {
            v = ((v & 63u) | (v << 8)) & 0x300fu;
            v = (v | (v << 4)) & 0x30c3u;
            return (v | (v << 2)) & 0x9249u;
        };
        low = (low << 18) | spread(X) | (spread(Y) << 1) | (spread(Z) << 2);
    }
    const u64 xy = (u64)(X >> 7) + (u64)(Y >> 7) * (u32)kp.nx;
    if (z >= 0) return ((xy + (Z >> 7) * kp.nxy) << 21) | low;
    return kp.defect_flag | (xy << 21) | low;  // id = xy + defect_base
}

// Block keys from int32 lattice cells: those that the quantization sweep kept, or a cell table's
// (encode_cells_with_counts, composer/block_compressor_rle.hpp:341-470), for which
// cells_stats_kernel takes the per-axis minima / maxima.  Bound by instructions and by the histograms'
// shared atomics: one Hilbert level per read, 64-bit arithmetic and 4-byte loads took 218 instructions
// per key and 505 us for 64M; this 330, 3.9 TB/s.
template <bool VEC>
__global__ void __launch_bounds__(kThreads) keys_cells_kernel(const i32* __restrict__ cells, u64 n, BlockKeyParams kp,
                                                              const unsigned short* __restrict__ tab2_g,
                                                              unsigned long long* __restrict__ keys,
                                                              u32* __restrict__ payload, int passes, u32* hist) {
    __shared__ __align__(16) unsigned short tab2[2048];
    __shared__ u32 sh[8 * 256];
    reinterpret_cast<uint4*>(tab2)[threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(tab2_g) + threadIdx.x);
    for (int i = threadIdx.x; i < passes * 256; i += kThreads) sh[i] = 0;
    __syncthreads();
    DigitHist dh{sh, passes};
    const u64 stride = (u64)gridDim.x * kThreads, k0 = (u64)blockIdx.x * kThreads + threadIdx.x;
    u64 done = 0;
    if (VEC) {
        done = n / 4 * 4;
        for (u64 k = k0; k < n / 4; k += stride) {
            const int4* src = reinterpret_cast<const int4*>(cells) + 3 * k;
            const int4 v0 = __ldg(src), v1 = __ldg(src + 1), v2 = __ldg(src + 2);
            const u64 q[4] = {block_key(v0.x, v0.y, v0.z, kp, tab2), block_key(v0.w, v1.x, v1.y, kp, tab2),
                              block_key(v1.z, v1.w, v2.x, kp, tab2), block_key(v2.y, v2.z, v2.w, kp, tab2)};
            ulonglong2* dst = reinterpret_cast<ulonglong2*>(keys) + 2 * k;
            dst[0] = make_ulonglong2(q[0], q[1]);
            dst[1] = make_ulonglong2(q[2], q[3]);
            if (payload) {
                const u32 i = (u32)(4 * k);
                reinterpret_cast<uint4*>(payload)[k] = make_uint4(i, i + 1, i + 2, i + 3);
            }
            if (passes) {
#pragma unroll
                for (int j = 0; j < 4; ++j) dh.add(q[j]);
            }
        }
    }
    for (u64 i = done + k0; i < n; i += stride) {
        const u64 k = block_key(__ldg(cells + 3 * i), __ldg(cells + 3 * i + 1), __ldg(cells + 3 * i + 2), kp, tab2);
        keys[i] = k;
        if (payload) payload[i] = (u32)i;
        if (passes) dh.add(k);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kThreads)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

__global__ void __launch_bounds__(kThreads) cells_stats_kernel(const i32* __restrict__ cells, u64 n,
                                                               PointStats* stats) {
    i32 lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    const u64 stride = (u64)gridDim.x * kThreads;
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride)
        for (int a = 0; a < 3; ++a) {
            const i32 v = __ldg(cells + 3 * i + a);
            lo[a] = min(lo[a], v);
            hi[a] = max(hi[a], v);
        }
    for (int a = 0; a < 3; ++a) {
        for (int d = 16; d > 0; d >>= 1) {
            lo[a] = min(lo[a], __shfl_xor_sync(kFullMask, lo[a], d));
            hi[a] = max(hi[a], __shfl_xor_sync(kFullMask, hi[a], d));
        }
        if (lane_id() == 0) {
            atomicMin(&stats->min_cell[a], lo[a]);
            atomicMax(&stats->max_cell[a], hi[a]);
        }
    }
}

__global__ void gather_i32_kernel(const i32* __restrict__ src, const u32* __restrict__ idx, u64 n,
                                  i32* __restrict__ dst) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        dst[i] = src[idx[i]];
}

// expand_cells_to_points (composer/block_decompressor_rle.hpp:339-358): every cell repeated
// counts[i] times, recovered and unshifted; output positions by a chained scan of the counts.
__global__ void __launch_bounds__(kThreads) expand_cells_kernel(const i32* __restrict__ cells,
                                                                const i32* __restrict__ counts, u64 n, QuantParams q,
                                                                const float* __restrict__ off3, ScanStatus status,
                                                                u32* tile_counter, float* __restrict__ out, u64 cap,
                                                                unsigned long long* total, u32* err) {
    constexpr int kItems = 16, kTile = kThreads * kItems;
    __shared__ u64 scratch[16];
    __shared__ u32 slot;
    __shared__ u64 sbase;
    const u32 tile = claim_tile(tile_counter, &slot);
    const u64 base = (u64)tile * kTile + (u64)threadIdx.x * kItems;
    u64 s = 0;
    for (int i = 0; i < kItems; ++i)
        if (base + i < n) s += (u64)max(__ldg(counts + base + i), 0);
    u64 tot;
    const u64 ex = block_exclusive<kThreads>(s, 0ull, AddOp{}, scratch, tot);
    if (threadIdx.x < 32) {
        const u64 r = chain_add(status, tile, tot, err);
        if (threadIdx.x == 0) {
            sbase = r;
            if (tile == gridDim.x - 1) *total = r + tot;
        }
    }
    __syncthreads();
    u64 pos = sbase + ex;
    const float ox = off3[0], oy = off3[1], oz = off3[2];
    for (int i = 0; i < kItems; ++i) {
        const u64 j = base + i;
        if (j >= n) break;
        const u64 c = (u64)max(__ldg(counts + j), 0);
        if (pos + c > cap) {
            atomicOr(err, kErrOverflow);
            break;
        }
        float x, y, z;
        recover(q, __ldg(cells + 3 * j), __ldg(cells + 3 * j + 1), __ldg(cells + 3 * j + 2), ox, oy, oz, x, y, z);
        for (u64 r = 0; r < c; ++r) {
            out[3 * (pos + r)] = x;
            out[3 * (pos + r) + 1] = y;
            out[3 * (pos + r) + 2] = z;
        }
        pos += c;
    }
}

// Direct mode: key = global Morton or Hilbert code (hilbert_bits levels); z == -1 cells keep
// their transformed low levels under defect_flag.
__global__ void __launch_bounds__(kThreads) keys_direct_kernel(const float* __restrict__ xyz, u64 n, QuantParams q,
                                                               const PointStats* stats, DirectKeyParams kp,
                                                               const u8* __restrict__ htab_g,
                                                               unsigned long long* __restrict__ keys,
                                                               u32* __restrict__ payload, int passes, u32* hist) {
    __shared__ float off[3];
    __shared__ u8 htab[256];
    __shared__ u32 sh[8 * 256];
    if (threadIdx.x == 0) load_offset(xyz, stats, off);
    stage_hilbert_table(htab_g, htab);
    for (int i = threadIdx.x; i < passes * 256; i += kThreads) sh[i] = 0;
    __syncthreads();
    DigitHist dh{sh, passes};
    for_each_point<4>(xyz, n, [&](u64 i, float fx, float fy, float fz) {
        const float px = __fsub_rn(fx, off[0]), py = __fsub_rn(fy, off[1]), pz = __fsub_rn(fz, off[2]);
        i32 x, y, z;
        quantize(q, px, py, pz, x, y, z);
        u64 m = morton3(x, y, z);
        if (kp.hilbert) m = hilbert_apply(htab, m, kp.bits, 0u);
        const u64 k = (z >= 0) ? m : (kp.defect_flag | (m & (kp.defect_flag - 1)));
        keys[i] = k;
        if (payload) payload[i] = (u32)i;
        if (passes) dh.add(k);
    });
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kThreads)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

__global__ void __launch_bounds__(kThreads) quantize_cells_kernel(const float* __restrict__ xyz, u64 n, QuantParams q,
                                                                  const PointStats* stats, i32* __restrict__ cells) {
    __shared__ float off[3];
    if (threadIdx.x == 0) load_offset(xyz, stats, off);
    __syncthreads();
    const u64 stride = (u64)gridDim.x * kThreads;
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride) {
        const float px = __fsub_rn(xyz[3 * i], off[0]);
        const float py = __fsub_rn(xyz[3 * i + 1], off[1]);
        const float pz = __fsub_rn(xyz[3 * i + 2], off[2]);
        quantize(q, px, py, pz, cells[3 * i], cells[3 * i + 1], cells[3 * i + 2]);
    }
}

__global__ void __launch_bounds__(kThreads) recover_cells_kernel(const i32* __restrict__ cells, u64 n, QuantParams q,
                                                                 const float* __restrict__ off,
                                                                 float* __restrict__ xyz) {
    const u64 stride = (u64)gridDim.x * kThreads;
    const float ox = off[0], oy = off[1], oz = off[2];
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride) {
        float x, y, z;
        recover(q, cells[3 * i], cells[3 * i + 1], cells[3 * i + 2], ox, oy, oz, x, y, z);
        xyz[3 * i] = x;
        xyz[3 * i + 1] = y;
        xyz[3 * i + 2] = z;
    }
}

__global__ void __launch_bounds__(kThreads) hilbert_kernel(const unsigned long long* __restrict__ in, u64 n,
                                                           const u8* __restrict__ tab_g, int top, u32 state,
                                                           unsigned long long* __restrict__ out) {
    __shared__ u8 tab[256];
    stage_hilbert_table(tab_g, tab);
    __syncthreads();
    const u64 stride = (u64)gridDim.x * kThreads;
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride) out[i] = hilbert_apply(tab, in[i], top, state);
}

int grid_for(u64 n) {
    // Persistent-style grid: a few resident blocks per SM of the 148-SM B200.
    u64 want = (n + kThreads - 1) / kThreads;
    u64 cap = 148ull * 8ull;
    if (want < 1) want = 1;
    return (int)(want < cap ? want : cap);
}

}  // namespace

void launch_bbox(const float* xyz, uint64_t n, PointStats* stats, cudaStream_t st) {
    // (four pieces per thread and loop; a multiple of three blocks)
    if (use_vec(n, xyz)) bbox_vec_kernel<<<(grid_for(3 * n / 16) + 2) / 3 * 3, kThreads, 0, st>>>(xyz, n, stats);
    else bbox_kernel<<<grid_for(n), kThreads, 0, st>>>(xyz, n, stats);
}
void launch_adaptive_steps(const float* xyz, float l2, PointStats* stats, cudaStream_t st) {
    adaptive_steps_kernel<<<1, 32, 0, st>>>(xyz, l2, stats);
}
void launch_quantize_range(const float* xyz, uint64_t n, QuantParams q, PointStats* stats, int with_error_stats,
                           cudaStream_t st, int32_t* cells) {
    if (use_vec(n, xyz, cells))
        quantize_range_kernel<true><<<grid_for(n / 4), kThreads, 0, st>>>(xyz, n, q, stats, with_error_stats, cells);
    else
        quantize_range_kernel<false><<<grid_for(n), kThreads, 0, st>>>(xyz, n, q, stats, with_error_stats, cells);
}
void launch_keys_direct(const float* xyz, uint64_t n, QuantParams q, const PointStats* stats, DirectKeyParams kp,
                        const uint8_t* hilbert_tab, unsigned long long* keys, uint32_t* payload, int passes,
                        uint32_t* hist, cudaStream_t st) {
    keys_direct_kernel<<<grid_for(n), kThreads, 0, st>>>(xyz, n, q, stats, kp, hilbert_tab, keys, payload, passes,
                                                         hist);
}
void launch_keys_cells(const int32_t* cells, uint64_t n, BlockKeyParams kp, const uint16_t* hilbert_fwd2,
                       unsigned long long* keys, uint32_t* payload, int passes, uint32_t* hist, cudaStream_t st) {
    // (keys and payload are the library's own buffers, aligned)
    if (use_vec(n, cells))
        keys_cells_kernel<true><<<grid_for(n / 4), kThreads, 0, st>>>(cells, n, kp, hilbert_fwd2, keys, payload, passes, hist);
    else
        keys_cells_kernel<false><<<grid_for(n), kThreads, 0, st>>>(cells, n, kp, hilbert_fwd2, keys, payload, passes, hist);
}
void launch_cells_stats(const int32_t* cells, uint64_t n, PointStats* stats, cudaStream_t st) {
    cells_stats_kernel<<<grid_for(n), kThreads, 0, st>>>(cells, n, stats);
}
void launch_gather_i32(const int32_t* src, const uint32_t* idx, uint64_t n, int32_t* dst, cudaStream_t st) {
    if (n) gather_i32_kernel<<<grid_for(n), kThreads, 0, st>>>(src, idx, n, dst);
}
void launch_expand_cells(const int32_t* cells, const int32_t* counts, uint64_t n, QuantParams q, const float* off3,
                         ScanStatus status, uint32_t* tile_counter, float* out, uint64_t cap,
                         unsigned long long* total, uint32_t* err, cudaStream_t st) {
    const unsigned tiles = (unsigned)((n + kThreads * 16 - 1) / (kThreads * 16));
    if (tiles) expand_cells_kernel<<<tiles, kThreads, 0, st>>>(cells, counts, n, q, off3, status, tile_counter, out, cap, total, err);
}
void launch_quantize_cells(const float* xyz, uint64_t n, QuantParams q, const PointStats* stats, int32_t* cells,
                           cudaStream_t st) {
    quantize_cells_kernel<<<grid_for(n), kThreads, 0, st>>>(xyz, n, q, stats, cells);
}
void launch_recover_cells(const int32_t* cells, uint64_t n, QuantParams q, const float* offset3_dev, float* xyz,
                          cudaStream_t st) {
    recover_cells_kernel<<<grid_for(n), kThreads, 0, st>>>(cells, n, q, offset3_dev, xyz);
}
void launch_hilbert(const unsigned long long* in, uint64_t n, const uint8_t* tab, int top, unsigned int state,
                    unsigned long long* out, cudaStream_t st) {
    hilbert_kernel<<<grid_for(n), kThreads, 0, st>>>(in, n, tab, top, state, out);
}

}  // namespace dev
}  // namespace xnyz
