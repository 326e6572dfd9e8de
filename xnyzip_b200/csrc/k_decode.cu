// Decompress-side kernels.
//
//   block_streams  BitPacker<uint64_t>::unpack (encoder/bitpacking_encoder.hpp:53-80) of the
//                  block-id and block-count deltas fused with their prefix sums
//                  (block_decompressor.hpp:159-161, u64, wrapping) and the block-start marks
//   (the entropy-coded streams are decoded in k_stream_decode.cu)
//   recover_units  recover_from_lcp_meta (block_quantizer.hpp:154-207) fused with the PFor
//                  decode, the direct-mode SFC prefix sum (block_decompressor.hpp:86-102), the
//                  -rle expansion (block_decompressor_rle.hpp:182-187), recover and unshift.
#include "device_common.cuh"
#include "kernels.h"

namespace xnyz {
namespace dev {

namespace {

constexpr int kThreads = 256;
// x / d for an invariant divisor (U64Div, kernels.h)
__device__ __forceinline__ u64 udiv(u64 x, const U64Div& d) {
    if (x < (1ull << 44)) return __umul64hi(x << 20, d.m44) >> d.l44;
    const u64 t = __umul64hi(d.m, x);
    return (t + ((x - t) >> d.sh1)) >> d.sh2;
}

// ------------------------------------------------------------- block streams -----------
// The -normal/-rle block streams of block mode in one pass (block_decompressor.hpp:111-161):
// bit-unpack the block-id deltas and block-count deltas, inclusive prefix sums of both
// (u64, wrapping), the exclusive prefix of the counts (first unit of each block), the per-unit
// block-start marks of recover_from_lcp_meta (block_quantizer.hpp:167-176), and the lattice corner
// of each block that has units (empty ones are skipped, as the reference does, so that block k of
// the output starts at the k-th mark).
//
// A tile is 2048 blocks.  Its packed words are staged in shared memory with all loads in flight, the
// thread that owns eight consecutive blocks unpacks and sums them in registers, one chained scan gives
// the tile's carries, and the outputs leave one block per lane.  The chain carries the ids' sum and,
// for the counts, (A, B) = the sum of the deltas and the sum of the counts, which from count carry 0 add
// up as (A1 + A2, B1 + B2 + N2 * A1) for N2 blocks (all but the last tile have 2048).  What bounds it:
// the latency of the loads and of the chain.  Rounds of warp scans over 32 blocks, unpacked twice, took
// 1054 us for 64M blocks, values one per lane from global memory with two chains 1282, this 910 (20
// and 12 us for 1013 points; with the deltas kept in shared memory instead of registers 976).
//
// Encoders write no empty blocks, so block j is the output's j-th; a block without units sets *empty,
// and the caller runs the COMPACT variant, which ranks the others by a second chained scan.
constexpr int kStreamItems = 8;
constexpr int kStreamTile = kThreads * kStreamItems;
static_assert(kStreamTile == kBlockStreamTile, "tile size");
constexpr int kStreamPad = 4;  // words of alignment before a tile's first

__device__ __forceinline__ u32 skew16(u32 w) { return w + (w >> 4); }
__device__ __forceinline__ u32 skew8(u32 e) { return e + (e >> 3); }  // a thread's eight values, two-way conflicts at most

// Ids' sum, deltas' sum, counts' sum, through two status words per tile: (ids, B's high half) and
// (A, B's low half); a pair seen between its two stores does not agree on the flag and counts as empty.
struct StreamSums {
    u64 id, a, b;
};
__device__ __forceinline__ void st_sums(Status* p, StreamSums v, u32 flag) {
    st_status(p, Pair{v.id, v.b >> 32}, flag);
    st_status(p + 1, Pair{v.a, v.b & 0xffffffffull}, flag);
}
__device__ __forceinline__ StreamSums ld_sums(const Status* p, u32& flag) {
    u32 f0, f1;
    const Pair x = ld_status(p, f0), y = ld_status(p + 1, f1);
    flag = f0 == f1 ? f0 : 0u;
    return StreamSums{x.lo, y.lo, (x.hi << 32) | y.hi};
}

// chain_lookback for StreamSums, two tiles per lane.
__device__ StreamSums streams_lookback(Status* status, u32 tile, StreamSums mine, u64 blocks, u32* err) {
    const int lane = (int)(threadIdx.x & 31u);
    if (lane == 0) st_sums(status + 2 * (u64)tile, mine, tile == 0 ? 2u : 1u);
    StreamSums acc{0, 0, 0};
    if (tile == 0) return acc;
    u64 after = 0;  // blocks between the window and the tile
    i64 top = (i64)tile - 1;
    u32 spins = 0;
    bool failed = false;
    while (true) {
        u32 f[2] = {2u, 2u};
        StreamSums v[2] = {};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const i64 q = top - 2 * lane - j;
            if (q >= 0) v[j] = ld_sums(status + 2 * q, f[j]);
        }
        const bool fin = f[0] == 2u || (f[0] && f[1] == 2u);
        const bool empty = f[0] == 0u || (f[0] != 2u && f[1] == 0u);
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
        // my tiles joined, then the lanes: earlier tiles first; d tiles hold kStreamTile blocks each
        StreamSums r = v[0];
        if (f[0] != 2u) {
            r.b = v[1].b + r.b + (u64)kStreamTile * v[1].a;
            r.a += v[1].a;
            r.id += v[1].id;
        }
        if (lane > last) r = StreamSums{0, 0, 0};
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const StreamSums o{__shfl_down_sync(kFullMask, r.id, d), __shfl_down_sync(kFullMask, r.a, d),
                               __shfl_down_sync(kFullMask, r.b, d)};
            if (lane + d < 32) {  // r covers 2 d tiles, all of them before the last one of the stream
                r.b = o.b + r.b + (u64)(2 * d) * kStreamTile * o.a;
                r.a += o.a;
                r.id += o.id;
            }
        }
        const StreamSums w{__shfl_sync(kFullMask, r.id, 0), __shfl_sync(kFullMask, r.a, 0), __shfl_sync(kFullMask, r.b, 0)};
        acc.b = w.b + acc.b + after * w.a;
        acc.a += w.a;
        acc.id += w.id;
        after += 64ull * kStreamTile;
        if (m2) break;
        top -= 64;
    }
    if (lane == 0) {
        if (failed) atomicOr(err, kErrTimeout);
        st_sums(status + 2 * (u64)tile, StreamSums{acc.id + mine.id, acc.a + mine.a, acc.b + mine.b + blocks * acc.a}, 2u);
    }
    return acc;
}

template <bool COMPACT>
__global__ void __launch_bounds__(kThreads, 4) block_streams_kernel(const u32* __restrict__ wb, u64 bb, int width_b,
                                                                 const u32* __restrict__ wc, u64 bc, int width_c,
                                                                 u64 nb, u64 units, U64Div div_nx, U64Div div_ny,
                                                                 u32 nx, u32 ny, BlockCorners corners,
                                                                 u8* __restrict__ is_start, Status* status,
                                                                 u32* tile_counter, unsigned long long* count_total,
                                                                 u32* empty, u32* err) {
    constexpr int kW = kThreads / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ u64 wid[kW], wcnt[kW], wsum[kW];  // per warp: totals, then prefixes
    __shared__ u32 wrank[kW];
    __shared__ u64 first_carry;
    __shared__ u64 first_rank;
    __shared__ u32 slot;
    const u32 tile = claim_tile(tile_counter, &slot);
    const int tid = threadIdx.x, w = tid >> 5;
    const u32 lane = lane_id();
    const u64 base = (u64)tile * kStreamTile;
    const u32 have = (u32)min((u64)kStreamTile, nb - base);
    const u32 e0 = (u32)tid * kStreamItems;
    // the tile's words of one stream, from a 16-byte boundary on; returns the bit of its first value
    auto stage = [&](const u32* __restrict__ words, u64 bit0, int width, u32* s) -> u32 {
        const u64 at = bit0 + base * (u64)width;
        const u32* p = words + (at >> 5);
        const u32 lead = (u32)(reinterpret_cast<uintptr_t>(p) & 15u) / 4u;
        const u32 n = (lead + (((u32)at & 31u) + have * (u32)width + 31u) / 32u + 2u + 3u) / 4u;  // (+ a value's spare words)
        const uint4* v = reinterpret_cast<const uint4*>(p - lead);
#pragma unroll 8
        for (u32 i = tid; i < n; i += kThreads) {
            const uint4 q = __ldg(v + i);
            s[skew16(4 * i)] = q.x;
            s[skew16(4 * i + 1)] = q.y;
            s[skew16(4 * i + 2)] = q.z;
            s[skew16(4 * i + 3)] = q.w;
        }
        return lead * 32u + ((u32)at & 31u);
    };
    auto unpack = [&](const u32* s, u32 q0, int width, u64 (&v)[kStreamItems]) {
        const u32 mlo = width >= 32 ? ~0u : ((1u << width) - 1u), mhi = width >= 64 ? ~0u : width > 32 ? ((1u << (width - 32)) - 1u) : 0u;
#pragma unroll
        for (int i = 0; i < kStreamItems; ++i) {
            v[i] = 0;
            if (e0 + i < have && width) {
                const u32 q = q0 + (e0 + i) * (u32)width, x = q >> 5;
                const u32 x1 = s[skew16(x + 1)];
                const u32 lo = __funnelshift_r(s[skew16(x)], x1, q) & mlo;
                const u32 hi = width > 32 ? __funnelshift_r(x1, s[skew16(x + 2)], q) & mhi : 0u;
                v[i] = (u64)lo | ((u64)hi << 32);
            }
        }
    };
    u32* sw = reinterpret_cast<u32*>(smem_raw);
    u32* sw1 = sw + skew16((u32)(kStreamTile / 32 * width_b) + 4 + kStreamPad + 4);
    const u32 qb = stage(wb, bb, width_b, sw), qc = stage(wc, bc, width_c, sw1);
    __syncthreads();
    u64 db[kStreamItems], dc[kStreamItems];
    unpack(sw, qb, width_b, db);
    unpack(sw1, qc, width_c, dc);
    // sums of the ids and of the count deltas; S: sum of the counts from count carry 0
    u64 id = 0, cnt = 0, sum = 0;
    const u32 mine = e0 < have ? min(have - e0, (u32)kStreamItems) : 0u;
#pragma unroll
    for (int i = 0; i < kStreamItems; ++i) {
        id += db[i];
        cnt += dc[i];
        if (i < (int)mine) sum += cnt;
    }
    {
        const u64 i1 = warp_incl_add(id), c1 = warp_incl_add(cnt);
        const u64 s1 = warp_incl_add(sum + (u64)mine * (c1 - cnt));  // from the warp's carry 0
        if (lane == 31) {
            wid[w] = i1;
            wcnt[w] = c1;
            wsum[w] = s1;
        }
        id = i1 - id;
        sum = s1 - (sum + (u64)mine * (c1 - cnt));
        cnt = c1 - cnt;
    }
    __syncthreads();
    if (w == 0) {
        const u32 wm = lane < kW && lane * 256u < have ? min(have - lane * 256u, 256u) : 0u;  // the warp's blocks
        const u64 x = lane < kW ? wid[lane] : 0ull, xi = warp_incl_add(x);
        const u64 y = lane < kW ? wcnt[lane] : 0ull, yi = warp_incl_add(y);
        const u64 z = (lane < kW ? wsum[lane] : 0ull) + (u64)wm * (yi - y), zi = warp_incl_add(z);
        const StreamSums total{__shfl_sync(kFullMask, xi, 31), __shfl_sync(kFullMask, yi, 31), __shfl_sync(kFullMask, zi, 31)};
        const StreamSums r = streams_lookback(status, tile, total, have, err);
        if (lane < kW) {
            wid[lane] = r.id + xi - x;
            wcnt[lane] = r.a + yi - y;
            wsum[lane] = r.b + zi - z;  // but for the tile's count carry
        }
        if (lane == 0) {
            first_carry = r.a;
            if (tile == gridDim.x - 1) *count_total = r.b + total.b + have * r.a;
        }
    }
    __syncthreads();
    const u64 carry = first_carry;  // count before the tile
    // my blocks' ids, first units and ranks, to shared memory
    u64* sid = reinterpret_cast<u64*>(smem_raw);                   // kStreamTile, skewed by one per 8
    u32* sstart = reinterpret_cast<u32*>(sid + kStreamTile + kStreamTile / 8);
    unsigned short* srank = reinterpret_cast<unsigned short*>(sstart + kStreamTile + kStreamTile / 8);
    const u32 s0 = skew8(e0);
    // blocks before mine in my warp count wcnt[w] - carry more each than from the warp's carry 0
    const u32 before_lane = min(lane * (u32)kStreamItems, have > (u32)w * 256u ? have - (u32)w * 256u : 0u);
    u64 start = sum + (u64)before_lane * (wcnt[w] - carry) + wsum[w] + carry * (u64)min(e0, have);
    id += wid[w];
    cnt += wcnt[w];
    u32 rank = 0;
    if (COMPACT) {
        u64 c = cnt;
        u32 n = 0;
#pragma unroll
        for (int i = 0; i < kStreamItems; ++i) {
            c += dc[i];
            n += i < (int)mine && c > 0;
        }
        const u32 r1 = warp_incl_add(n);
        if (lane == 31) wrank[w] = r1;
        rank = r1 - n;
        __syncthreads();
        if (w == 0) {
            const u32 y = lane < kW ? wrank[lane] : 0u, yi = warp_incl_add(y);
            const u64 r = chain_add(status + 2 * (u64)gridDim.x, tile, __shfl_sync(kFullMask, yi, 31), err);
            if (lane < kW) wrank[lane] = yi - y;
            if (lane == 0) first_rank = r;
        }
        __syncthreads();
        rank += wrank[w];
    } else {
        rank = e0;
    }
    bool none = false;
#pragma unroll
    for (int i = 0; i < kStreamItems; ++i) {
        id += db[i];
        cnt += dc[i];
        sid[s0 + i] = id;
        sstart[s0 + i] = start < units ? (u32)start : 0xffffffffu;  // (units are below 2^32 - 1)
        const bool filled = i < (int)mine && cnt > 0;
        none |= i < (int)mine && cnt == 0;
        srank[e0 + i] = filled ? (unsigned short)rank : (unsigned short)0xffffu;
        rank += COMPACT ? (u32)filled : 1u;
        start += cnt;
    }
    if (!COMPACT && none) atomicOr(empty, 1u);
    __syncthreads();
    const u64 r0 = COMPACT ? first_rank : base;
    u32 *cx = corners.x + r0, *cy = corners.y + r0, *cz = corners.z + r0;
#pragma unroll 4
    for (int i = 0; i < kStreamItems; ++i) {
        const u32 e = (u32)i * kThreads + tid;
        const u32 rk = srank[e], su = sstart[skew8(e)];
        if (rk == 0xffffu || su == 0xffffffffu) continue;
        is_start[su] = 1;
        const u64 blk = sid[skew8(e)], q1 = udiv(blk, div_nx), q2 = udiv(q1, div_ny);
        // ((blk % nx) * 128, (blk / nx % ny) * 128, (blk / nx / ny) * 128) in u64 arithmetic, kept modulo
        // 2^32 like the cell coordinates they are added to
        cx[rk] = ((u32)blk - (u32)q1 * nx) * 128u;
        cy[rk] = ((u32)q1 - (u32)q2 * ny) * 128u;
        cz[rk] = (u32)q2 * 128u;
    }
}

size_t block_streams_smem(int width_b, int width_c) {
    auto words = [](int width) { const u32 n = (u32)(kStreamTile / 32 * width) + 4 + kStreamPad + 4; return (size_t)(n + (n >> 4)); };
    const size_t staged = 4 * (words(width_b) + words(width_c) + 8);
    const size_t out = (kStreamTile + kStreamTile / 8) * 12 + kStreamTile * 2;
    return staged > out ? staged : out;
}

// ------------------------------------------------------------- tile prefixes -----------
// Per tile of 2048 units: how many patches, block starts and outputs come before it, by one chained
// scan over groups of four tiles, so that recover_units need not wait for three.  Bound by memory when
// large: 130 us for 64M units (6 bytes each), 3 TB/s; by latency for 1M units, 15 us (17 in groups of eight).
__global__ void __launch_bounds__(kThreads) tile_prefix_kernel(const u8* __restrict__ rep_sym, const u8* __restrict__ is_start,
                                                               const i32* __restrict__ counts, u64 units, TilePrefix* out,
                                                               Status* status, u32* tile_counter,
                                                               unsigned long long* count_total, u32* err) {
    constexpr int kW = kThreads / 32;
    __shared__ u32 sz[kPrefixTiles][kW], ss[kPrefixTiles][kW];
    __shared__ u64 sc[kPrefixTiles][kW];
    __shared__ u32 slot;
    const u32 group = claim_tile(tile_counter, &slot);
    const int tid = threadIdx.x, w = tid >> 5;
    const u32 lane = lane_id();
#pragma unroll
    for (int g = 0; g < kPrefixTiles; ++g) {
        const u64 e0 = ((u64)group * kPrefixTiles + g) * kRecoverTile + (u32)tid * 8u;
        const u32 have = e0 < units ? (u32)min(units - e0, (u64)8) : 0u;
        const u64 keep = have >= 8u ? ~0ull : ((1ull << (8 * have)) - 1);
        u32 z = 0, s = 0;
        u64 c = 0;
        if (have) {
            if (rep_sym) {
                const u64 r = __ldg(reinterpret_cast<const u64*>(rep_sym + e0)) | ~keep;
                z = (u32)(__popc(__vcmpeq4((u32)r, 0u)) + __popc(__vcmpeq4((u32)(r >> 32), 0u))) / 8u;
            }
            if (is_start) s = (u32)__popcll(__ldg(reinterpret_cast<const u64*>(is_start + e0)) & keep);
            if (counts) {
                const int4 a = __ldg(reinterpret_cast<const int4*>(counts + e0));
                const int4 b = have > 4u ? __ldg(reinterpret_cast<const int4*>(counts + e0 + 4)) : make_int4(0, 0, 0, 0);
                const i32 x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) c += i < (int)have ? (u64)max(x[i], 0) : 0ull;
            }
        }
        z = warp_sum(z);
        s = warp_sum(s);
        c = warp_sum(c);
        if (lane == 0) {
            sz[g][w] = z;
            ss[g][w] = s;
            sc[g][w] = c;
        }
    }
    __syncthreads();
    if (w == 0) {
        Pair x{0, 0};  // lane g: patches | starts << 32, outputs of tile g
        if (lane < kPrefixTiles)
            for (int i = 0; i < kW; ++i) x = PairAdd{}(x, Pair{(u64)sz[lane][i] | ((u64)ss[lane][i] << 32), sc[lane][i]});
        const Pair incl{warp_incl_add(x.lo), warp_incl_add(x.hi)};
        const Pair total{__shfl_sync(kFullMask, incl.lo, 31), __shfl_sync(kFullMask, incl.hi, 31)};
        const Pair r = chain_lookback(status, group, total, PairAdd{}, err);
        const u64 t = (u64)group * kPrefixTiles + lane;
        if (lane < kPrefixTiles && t * kRecoverTile < units) {
            const u64 lo = r.lo + incl.lo - x.lo;
            out[t] = TilePrefix{(u32)lo, (u32)(lo >> 32), r.hi + incl.hi - x.hi};
        }
        if (lane == 0 && group == gridDim.x - 1) {
            *count_total = r.hi + total.hi;
            const u64 lo = r.lo + total.lo;
            out[(units + kRecoverTile - 1) / kRecoverTile] = TilePrefix{(u32)lo, (u32)(lo >> 32), r.hi + total.hi};
        }
    }
}

// ---------------------------------------------------------------- header --------------
// One block: thread 0 walks the streams' lengths (a chain of one read each), then all threads copy
// the pieces.
__global__ void __launch_bounds__(kThreads) header_kernel(const u8* __restrict__ c, u64 len, u64 magic, int rle,
                                                          u8* __restrict__ out) {
    __shared__ HeaderPieces hp;
    constexpr u32 kRoom = (u32)(kHeaderBytes - sizeof(HeaderPieces));
    if (threadIdx.x == 0) {
        auto u64_at = [&](u64 p) {
            u64 v = 0;
#pragma unroll
            for (int b = 0; b < 8; ++b) v |= (u64)__ldg(c + p + b) << (8 * b);
            return v;
        };
        u32 used = 0;
        hp.count = 0;
        hp.unused = 0;
        auto take = [&](u64 off, u64 n) {
            const u32 m = (u32)min(n, (u64)(kRoom - used));
            hp.piece[hp.count++] = {off, m, used};
            used += m;
        };
        u64 p = 0;
        bool ok = len >= 64;
        if (ok) {
            if (u64_at(0) == magic) p = 8;
            const u64 np = u64_at(p + 8);  // quantizer parameters (4 bytes each)
            p += 16;
            ok = np <= (len - p) / 4 && len - p - 4 * np >= 14;
            if (ok) {
                p += 4 * np + 13;
                const int ns = (__ldg(c + p) ? 2 : 6) + rle;  // the direct-mode flag ends the fixed fields
                ++p;
                u64 from = 0;  // a piece holds the fixed fields or nothing, a stream's lengths and its meta
                for (int i = 0; i < ns && ok; ++i) {
                    ok = len - p >= 16;
                    if (!ok) break;
                    const u64 dl = u64_at(p), ml = u64_at(p + 8);
                    p += 16;
                    ok = ml <= len - p && dl <= len - p - ml;
                    take(from, p - from + (ok ? ml : 0));
                    p += ok ? ml + dl : 0;
                    from = p;
                }
                if (ok && len - p >= 12) take(p, 12);
            }
        }
    }
    __syncthreads();
    u8* bytes = out + sizeof(HeaderPieces);
    for (u32 i = 0; i < hp.count; ++i)
        for (u32 b = threadIdx.x; b < hp.piece[i].len; b += kThreads)
            bytes[hp.piece[i].at + b] = __ldg(c + hp.piece[i].off + b);
    for (u32 b = threadIdx.x; b < sizeof(HeaderPieces) / 4; b += kThreads)
        reinterpret_cast<u32*>(out)[b] = reinterpret_cast<const u32*>(&hp)[b];
}

// ---------------------------------------------------------------- helpers --------------
__global__ void fill_u32_kernel(u32* p, u64 n, u32 v) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) p[i] = v;
}
__global__ void fill_u8_kernel(u8* p, u64 n, u8 v) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) p[i] = v;
}

// ------------------------------------------------------------- recover units -------------
struct RecoverArgs {
    const u8* rep_sym;
    const void* rep_patch;
    int patch32;
    u64 npatch;
    const u8* quad_sym;
    const u8* is_start;
    BlockCorners corners;
    u64 nblocks;
    const i32* counts;
    const u64* rep_val;
    u64 units;
    u64 nout;
    RecoverParams rp;
    const u8* hinv;
    const unsigned short* hinv2;
    const TilePrefix* prefix;  // per tile and one past the last
    Status* status;            // segments (block mode) or SFC sums
    u32* tile_counter;
    float* out;
    u32* err;
};

// Block mode's segmented sums, chained over the tiles.  lo: repos sum since the last repos head; hi: quad
// sum modulo 8 since the last block start (bits 32..34), whether a block starts (35) and whether a repos
// head is inside (36).  A tile with both is closed: the walk normally ends at the tile before.
struct SegPair {
    __device__ __forceinline__ Pair operator()(Pair a, Pair b) const {
        const bool hq = (b.hi >> 35) & 1u, hr = (b.hi >> 36) & 1u;
        const u64 quad = ((hq ? 0ull : a.hi >> 32) + (b.hi >> 32)) & 7u;
        return Pair{(hr ? 0ull : a.lo) + b.lo, (quad << 32) | ((a.hi | b.hi) & (3ull << 35))};
    }
    __device__ static __forceinline__ bool closed(Pair v) { return ((v.hi >> 35) & 3u) == 3u; }
};
constexpr u64 kSegQuad = 1ull << 35, kSegRep = 1ull << 36;

// recover + unshift (device_common.cuh: recover), the divisions by the constant as above when allowed;
// v * 2 * s is v * (2 s), doubling being exact.
__device__ __forceinline__ void recover_point(const RecoverParams& p, i32 cx, i32 cy, i32 cz, float& x, float& y,
                                              float& z) {
    if (!p.q.rinv || p.q.quantizer == 2) {
        recover(p.q, cx, cy, cz, p.off[0], p.off[1], p.off[2], x, y, z);
        return;
    }
    float f[3];
    if (p.q.quantizer == 1) {
        const u32 odd = (u32)cz & 1u;
        f[0] = __int2float_rn((i32)(((u32)cx << 1) - odd));
        f[1] = __int2float_rn((i32)(((u32)cy << 1) - odd));
        f[2] = __int2float_rn(cz);
    } else {
        f[0] = __fadd_rn(__int2float_rn(cx), 0.5f);
        f[1] = __fadd_rn(__int2float_rn(cy), 0.5f);
        f[2] = __fadd_rn(__int2float_rn(cz), 0.5f);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) f[a] = div_const(__fmul_rn(f[a], 2.0f * p.q.s), p.q.rdiv, p.q.rinv);
    x = __fadd_rn(f[0], p.off[0]);
    y = __fadd_rn(f[1], p.off[1]);
    z = __fadd_rn(f[2], p.off[2]);
}

// Block mode's segmented sums within a tile.  rep: repos sum since the last head; m: block starts (bits
// 0..11), quad sum modulo 8 since the last start (16..18), a start (30) and a repos head (31) inside.
template <typename T>
struct TileSeg {
    T rep;
    u32 m;
};
template <typename T>
__device__ __forceinline__ TileSeg<T> seg_join(TileSeg<T> a, TileSeg<T> b) {
    const u32 quad = ((b.m & (1u << 30) ? 0u : a.m) + b.m) & (7u << 16);
    return TileSeg<T>{(T)((b.m >> 31 ? (T)0 : a.rep) + b.rep), ((a.m + b.m) & 0xfffu) | quad | ((a.m | b.m) & (3u << 30))};
}
template <typename T>
__device__ __forceinline__ TileSeg<T> seg_warp_incl(TileSeg<T> v) {
    const u32 lane = lane_id();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const TileSeg<T> o{__shfl_up_sync(kFullMask, v.rep, d), __shfl_up_sync(kFullMask, v.m, d)};
        if (lane >= (u32)d) v = seg_join(o, v);
    }
    return v;
}

// A tile is 2048 units.  Thread t owns units [8 t, 8 t + 8): it reads their symbols as one 8-byte
// word each and sums their values serially, which it keeps in its own slots of shared memory; one scan
// over the threads and one chained scan over the tiles (patches, counts and starts come from launch_tile_prefix) turn
// them into true carries, with which the thread writes each unit's repos code (or SFC), quad and block
// to shared memory.  The last phase takes one unit per lane: corners and points of neighbouring lanes
// are neighbours in memory.  What bounds it: instructions (the Hilbert digits, two levels per table
// read, and the three divisions, as multiplications by the reciprocal).  Rounds of warp scans over 32
// units took 1681 us for 64M units (block mode, Hilbert, -rle) and 47 us for 1013; this takes 875 and 16, and
// the prefixes 130 and 8 (three chained scans in here: 1443; the values in registers, so four blocks per SM
// instead of six: 1169).
constexpr int kRecItems = 8;
constexpr int kRecTile = kThreads * kRecItems;
static_assert(kRecTile == kRecoverTile, "tile size");
constexpr int kBatch = 2;  // units per lane computed before their points are written

struct RecoverShared {
    u64 rep[kRecTile + kRecTile / 8];        // values, then repos codes or SFCs, skewed
    u32 pos[kRecTile + kRecTile / 32 + 1];   // patches (one pad word per 32), then -rle output positions in the tile
    unsigned short meta[kRecTile];           // quad | block start number within the tile << 3
    u64 wrep[kThreads / 32], wcnt[kThreads / 32];
    u32 wm[kThreads / 32], wz[kThreads / 32];
    u64 rep0;
    u32 quad0;
};

// From the thread's values to the units' codes, quads, blocks and output positions in shared memory.
// T: the type of the tile's repos sums (u32 when every value is below 2^20).
template <bool DIRECT, typename T>
__device__ __forceinline__ void recover_scan(const RecoverArgs& a, RecoverShared& sh, u32 tile, u64 quads, u64 starts,
                                             u32 mine, bool rle) {
    constexpr int kW = kThreads / 32;
    const int tid = threadIdx.x, w = tid >> 5;
    const u32 lane = lane_id(), e0 = (u32)tid * kRecItems;
    u64* const v = sh.rep + skew8(e0);  // my values, in the end my codes
    // my counts (read twice rather than kept)
    auto counts = [&](u32 (&c)[kRecItems]) {
#pragma unroll
        for (int i = 0; i < kRecItems; i += 4) {
            const int4 q = i < (int)mine ? __ldg(reinterpret_cast<const int4*>(a.counts + (u64)tile * kRecTile + e0 + i))
                                         : make_int4(0, 0, 0, 0);
            const i32 x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) c[i + k] = i + k < (int)mine ? (u32)max(x[k], 0) : 0u;
        }
    };
    // unit i: quad step (0 for the patch symbol 0, which never occurs and is flagged) and heads
    auto unit = [&](int i) -> TileSeg<T> {
        const u32 q = (u32)(quads >> (8 * i)) & 255u, st = (u32)(starts >> (8 * i)) & 1u;
        const u32 step = q == 0u ? 0u : (q - 1u) & 7u;
        const bool head = i < (int)mine && (st || q != 1u);
        return TileSeg<T>{(T)v[i], st | (step << 16) | (st << 30) | (head ? 1u << 31 : 0u)};
    };
    TileSeg<T> agg{0, 0};
    u64 direct = 0, csum = 0;
#pragma unroll
    for (int i = 0; i < kRecItems; ++i) {
        if (DIRECT) direct += v[i];
        else agg = seg_join(agg, unit(i));
    }
    u64 cincl = 0;
    if (rle) {
        u32 c[kRecItems];
        counts(c);
#pragma unroll
        for (int i = 0; i < kRecItems; ++i) csum += c[i];
        cincl = warp_incl_add(csum);
        if (lane == 31) sh.wcnt[w] = cincl;
    }
    TileSeg<T> pre{0, 0};
    u64 dpre = 0;
    if (DIRECT) {
        const u64 incl = warp_incl_add(direct);
        if (lane == 31) sh.wrep[w] = incl;
        dpre = incl - direct;
    } else {
        const TileSeg<T> incl = seg_warp_incl(agg);
        if (lane == 31) {
            sh.wrep[w] = incl.rep;
            sh.wm[w] = incl.m;
        }
        pre = TileSeg<T>{__shfl_up_sync(kFullMask, incl.rep, 1), __shfl_up_sync(kFullMask, incl.m, 1)};
        if (lane == 0) pre = TileSeg<T>{0, 0};
    }
    __syncthreads();
    // the warps' totals become prefixes within the tile; the tile's total is chained
    if (w == 0) {
        Status* st = a.status;
        if (DIRECT) {
            const u64 x = lane < kW ? sh.wrep[lane] : 0ull, incl = warp_incl_add(x);
            const u64 r = chain_add(st, tile, __shfl_sync(kFullMask, incl, 31), a.err);
            if (lane < kW) sh.wrep[lane] = incl - x;
            if (lane == 0) sh.rep0 = r;
        } else {
            const TileSeg<T> x{lane < kW ? (T)sh.wrep[lane] : (T)0, lane < kW ? sh.wm[lane] : 0u};
            const TileSeg<T> incl = seg_warp_incl(x);
            const u64 trep = __shfl_sync(kFullMask, (u64)incl.rep, 31);
            const u32 tm = __shfl_sync(kFullMask, incl.m, 31);
            const Pair total{trep, ((u64)((tm >> 16) & 7u) << 32) | ((tm >> 30) & 1u ? kSegQuad : 0ull) |
                                       (tm >> 31 ? kSegRep : 0ull)};
            const Pair r = chain_lookback(st, tile, total, SegPair{}, a.err);
            TileSeg<T> ex{__shfl_up_sync(kFullMask, incl.rep, 1), __shfl_up_sync(kFullMask, incl.m, 1)};
            if (lane == 0) ex = TileSeg<T>{0, 0};
            if (lane < kW) {
                sh.wrep[lane] = ex.rep;
                sh.wm[lane] = ex.m;
            }
            if (lane == 0) {
                sh.rep0 = r.lo;
                sh.quad0 = (u32)(r.hi >> 32) & 7u;
            }
        }
    } else if (w == 1 && rle) {
        const u64 x = lane < kW ? sh.wcnt[lane] : 0ull, incl = warp_incl_add(x);
        if (lane < kW) sh.wcnt[lane] = incl - x;
    }
    __syncthreads();  // (also: every thread has its patches, pos and rep are free)
    if (DIRECT) {
        u64 run = sh.rep0 + sh.wrep[w] + dpre;
#pragma unroll
        for (int i = 0; i < kRecItems; ++i) {
            run += v[i];
            v[i] = run;
        }
    } else {
        TileSeg<T> run = seg_join(TileSeg<T>{(T)sh.wrep[w], sh.wm[w]}, pre);
        const u64 rep0 = sh.rep0;
        const u32 quad0 = sh.quad0;
        bool bad = false;
#pragma unroll
        for (int i = 0; i < kRecItems; ++i) {
            bad |= ((quads >> (8 * i)) & 255u) == 0u;
            run = seg_join(run, unit(i));
            v[i] = (run.m >> 31 ? 0ull : rep0) + run.rep;
            const u32 quad = ((run.m >> 16) + (run.m & (1u << 30) ? 0u : quad0)) & 7u;
            sh.meta[e0 + i] = (unsigned short)(quad | ((run.m & 0xfffu) << 3));
        }
        if (bad) atomicOr(a.err, kErrBadStream);
    }
    if (rle) {
        u64 pos = sh.wcnt[w] + cincl - csum;
        u32 c[kRecItems];
        counts(c);
#pragma unroll
        for (int i = 0; i < kRecItems; ++i) {
            sh.pos[e0 + i] = (u32)pos;
            pos += c[i];
        }
        if (tid == kThreads - 1) sh.pos[kRecTile] = (u32)pos;
    }
    __syncthreads();
}

template <bool DIRECT>
__global__ void __launch_bounds__(kThreads, 6) recover_units_kernel(const __grid_constant__ RecoverArgs a) {
    __shared__ RecoverShared sh;
    __shared__ __align__(16) unsigned short htab2[DIRECT ? 8 : 2048];  // two Hilbert levels per read
    __shared__ u8 htab[256];
    __shared__ u32 slot;
    const u32 tile = claim_tile(a.tile_counter, &slot);
    const u64 base = (u64)tile * kRecTile;
    const u32 cnt = (u32)min((u64)kRecTile, a.units - base);
    const int tid = threadIdx.x, w = tid >> 5;
    const u32 lane = lane_id(), e0 = (u32)tid * kRecItems;
    const bool has_val = a.rep_val != nullptr;
    const bool rle = a.rp.rle != 0;
    const TilePrefix pre = a.prefix[tile], next = a.prefix[tile + 1];
    htab[tid] = a.hinv[tid];
    if (!DIRECT) reinterpret_cast<uint4*>(htab2)[tid] = __ldg(reinterpret_cast<const uint4*>(a.hinv2) + tid);

    // my symbols: bytes past the end read as 1 (no patch, no step), no starts
    const u32 mine = e0 < cnt ? min(cnt - e0, 8u) : 0u;
    const u64 tail = mine >= 8u ? 0ull : ~0ull << (8 * mine);  // bytes past the end
    constexpr u64 kOnes = 0x0101010101010101ull;
    u64 reps = kOnes, quads = kOnes, starts = 0;
    if (mine) {
        if (!has_val) reps = (__ldg(reinterpret_cast<const u64*>(a.rep_sym + base + e0)) & ~tail) | (kOnes & tail);
        if (!DIRECT) {
            quads = (__ldg(reinterpret_cast<const u64*>(a.quad_sym + base + e0)) & ~tail) | (kOnes & tail);
            starts = __ldg(reinterpret_cast<const u64*>(a.is_start + base + e0)) & ~tail;
        }
    }
    u64* const v = sh.rep + skew8(e0);  // my values
    bool big = false;
    if (has_val) {
#pragma unroll
        for (int i = 0; i < kRecItems; ++i) {
            const u64 x = i < (int)mine ? __ldg(a.rep_val + base + e0 + i) : 0ull;
            big |= (x >> 20) != 0;
            v[i] = x;
        }
    } else {
        // ---- the tile's patches (32-bit ones through shared memory); each thread's number among them ----
        const u32 zeros = (u32)(__popc(__vcmpeq4((u32)reps, 0u)) + __popc(__vcmpeq4((u32)(reps >> 32), 0u))) / 8u;
        const u32 zi = warp_incl_add(zeros);
        if (lane == 31) sh.wz[w] = zi;
        const u64 z0 = pre.zeros;
        const u32 nz = next.zeros - pre.zeros;
        const u32 there = (u32)min((u64)nz, z0 < a.npatch ? a.npatch - z0 : 0ull);
        if (there < nz && tid == 0) atomicOr(a.err, kErrBadStream);
        const u64* p64 = static_cast<const u64*>(a.rep_patch) + z0;
        if (a.patch32) {
            const u32* p32 = static_cast<const u32*>(a.rep_patch) + z0;
#pragma unroll
            for (u32 i = 0; i < (u32)kRecItems; ++i) {
                const u32 p = i * kThreads + tid;
                if (p < nz) sh.pos[p + (p >> 5)] = p < there ? __ldg(p32 + p) : 0u;
            }
        }
        __syncthreads();
        u32 z = zi - zeros;
        for (int i = 0; i < w; ++i) z += sh.wz[i];
#pragma unroll
        for (int i = 0; i < kRecItems; ++i) {
            const u32 sym = (u32)(reps >> (8 * i)) & 255u;
            u64 x = sym - 1u;
            if (!sym) {
                x = a.patch32 ? (u64)sh.pos[z + (z >> 5)] : z < there ? __ldg(p64 + z) : 0ull;
                ++z;
            }
            big |= (x >> 20) != 0;
            v[i] = x;
        }
    }
    const bool any_big = __syncthreads_or(big);  // (every thread has its patches)
    if (DIRECT || any_big) recover_scan<DIRECT, u64>(a, sh, tile, quads, starts, mine, rle);
    else recover_scan<DIRECT, u32>(a, sh, tile, quads, starts, mine, rle);

    // ---- one unit per lane: coordinates, recover, unshift, expand ----
    const u64 o0 = rle ? pre.outputs : base;                     // the tile's first output
    const u64 no = rle ? next.outputs - pre.outputs : (u64)cnt;  // and how many it has
    if (!a.rp.cells && (no >= 0xffffffffull || o0 + no > a.nout)) {  // (only a damaged stream)
        if (tid == 0) atomicOr(a.err, kErrOverflow);
        return;
    }
    const u32 blk0 = DIRECT ? 0u : pre.starts;
    const u32 *px = a.corners.x + blk0, *py = a.corners.y + blk0, *pz = a.corners.z + blk0;
    const u32 nblk = (u32)min(a.nblocks - min((u64)blk0, a.nblocks), (u64)0xffffu);  // blocks from blk0 on
    float* out = a.out + 3 * o0;
    for (u32 i = 0; i < kRecTile && i < cnt; i += kBatch * kThreads) {
        float p[kBatch][3];
        u32 at[kBatch], end[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const u32 e = min(i + k * kThreads + tid, cnt - 1u);
            const u64 code = sh.rep[skew8(e)];
            u32 gx, gy, gz;
            if (DIRECT) {
                if (a.rp.hilbert) {
                    hilbert_xyz(htab, code, a.rp.bits, 0u, gx, gy, gz);
                } else {
                    gx = gather3(code);
                    gy = gather3(code >> 1);
                    gz = gather3(code >> 2);
                }
            } else {
                const u32 m = sh.meta[e];
                // block of the unit: the one before the starts counted so far (block 0 before any)
                const i32 b = max((i32)(m >> 3) - 1, blk0 ? -1 : 0);
                u32 cx = 0, cy = 0, cz = 0;
                if (b < (i32)nblk) {
                    cx = __ldg(px + b);
                    cy = __ldg(py + b);
                    cz = __ldg(pz + b);
                }
                if (!a.rp.hilbert) {
                    gx = gather3(code);
                    gy = gather3(code >> 1);
                    gz = gather3(code >> 2);
                } else if (code < (1ull << 18)) {
                    // the 6 levels of one 64^3 quadrant, two per read: entry = x, y, z digits | state << 6
                    u32 s = a.rp.hstart_inv << 6;
                    const u32 lo = (u32)code;
                    gx = gy = gz = 0;
#pragma unroll
                    for (int l = 2; l >= 0; --l) {
                        const u32 t = htab2[(s & ~63u) | ((lo >> (6 * l)) & 63u)];
                        gx = (gx << 2) | (t & 3u);
                        gy = (gy << 2) | ((t >> 2) & 3u);
                        gz = (gz << 2) | ((t >> 4) & 3u);
                        s = t;
                    }
                } else {
                    hilbert_xyz(htab, code, 20, 0u, gx, gy, gz);
                }
                gx += cx + (m & 1u) * 64u;
                gy += cy + ((m >> 1) & 1u) * 64u;
                gz += cz + ((m >> 2) & 1u) * 64u;
            }
            if (a.rp.cells) {
                p[k][0] = __int_as_float((i32)gx);
                p[k][1] = __int_as_float((i32)gy);
                p[k][2] = __int_as_float((i32)gz);
            } else {
                recover_point(a.rp, (i32)gx, (i32)gy, (i32)gz, p[k][0], p[k][1], p[k][2]);
            }
            // -rle: output position from the count prefix; -normal and cells: one per unit
            at[k] = rle ? sh.pos[e] : e;
            end[k] = i + k * kThreads + tid >= cnt ? 0u : rle ? sh.pos[e + 1] : e + 1u;
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
            for (u32 j = at[k]; j < end[k]; ++j) {
                float* o = out + 3ull * j;
                o[0] = p[k][0];
                o[1] = p[k][1];
                o[2] = p[k][2];
            }
    }
}

inline int grid_cap(u64 n) {
    u64 b = (n + kThreads - 1) / kThreads;
    if (b < 1) b = 1;
    return (int)(b < 148ull * 8 ? b : 148ull * 8);
}

}  // namespace

void launch_header(const uint8_t* cont, uint64_t len, int rle, uint8_t* out, cudaStream_t st) {
    header_kernel<<<1, kThreads, 0, st>>>(cont, len, kExtendedMagic, rle ? 1 : 0, out);
}
void launch_block_streams(const uint32_t* words_blk, uint64_t base_blk, int width_blk, const uint32_t* words_cnt,
                          uint64_t base_cnt, int width_cnt, uint64_t nblocks, uint64_t units, uint64_t nx, uint64_t ny,
                          bool compact, BlockCorners corners, uint8_t* is_start, ScanStatus status, uint32_t* tile_counter,
                          unsigned long long* count_total, uint32_t* empty, uint32_t* err, cudaStream_t st) {
    const unsigned tiles = (unsigned)((nblocks + kStreamTile - 1) / kStreamTile);
    if (!tiles) return;
    const size_t smem = block_streams_smem(width_blk, width_cnt);  // at most 37 KB
    auto k = compact ? block_streams_kernel<true> : block_streams_kernel<false>;
    k<<<tiles, kThreads, smem, st>>>(words_blk, base_blk, width_blk, words_cnt, base_cnt, width_cnt, nblocks, units,
                                     make_u64div(nx), make_u64div(ny), (u32)nx, (u32)ny, corners, is_start,
                                     static_cast<Status*>(status), tile_counter, count_total, empty, err);
}
void launch_tile_prefix(const uint8_t* rep_sym, const uint8_t* is_start, const int32_t* counts, uint64_t units,
                        TilePrefix* out, ScanStatus status, uint32_t* tile_counter, unsigned long long* count_total,
                        uint32_t* err, cudaStream_t st) {
    const u64 per = (u64)kRecoverTile * kPrefixTiles;
    const unsigned groups = (unsigned)((units + per - 1) / per);
    if (groups)
        tile_prefix_kernel<<<groups, kThreads, 0, st>>>(rep_sym, is_start, counts, units, out, static_cast<Status*>(status),
                                                        tile_counter, count_total, err);
}

void launch_fill_u32(uint32_t* p, uint64_t n, uint32_t v, cudaStream_t st) {
    if (n) fill_u32_kernel<<<grid_cap(n), kThreads, 0, st>>>(p, n, v);
}
void launch_fill_u8(uint8_t* p, uint64_t n, uint8_t v, cudaStream_t st) {
    if (n) fill_u8_kernel<<<grid_cap(n), kThreads, 0, st>>>(p, n, v);
}
void launch_recover_units(const RecoverInputs& in, uint64_t units, uint64_t nout, RecoverParams rp,
                          const uint8_t* hilbert_inv_tab, const uint16_t* hilbert_inv2, ScanStatus status, uint32_t* tile_counter, float* out, uint32_t* err,
                          cudaStream_t st) {
    RecoverArgs a;
    a.rep_sym = in.rep_sym;
    a.rep_patch = in.rep_patch;
    a.patch32 = in.patch32;
    a.npatch = in.npatch;
    a.quad_sym = in.quad_sym;
    a.is_start = in.is_start;
    a.corners = in.corners;
    a.nblocks = in.nblocks;
    a.counts = in.counts;
    a.rep_val = in.rep_val;
    a.units = units;
    a.nout = nout;
    a.rp = rp;
    a.hinv = hilbert_inv_tab;
    a.hinv2 = hilbert_inv2;
    a.prefix = in.prefix;
    a.status = static_cast<Status*>(status);
    a.tile_counter = tile_counter;
    a.out = out;
    a.err = err;
    const unsigned tiles = (unsigned)((units + kRecTile - 1) / kRecTile);
    if (!tiles) return;
    if (rp.direct)
        recover_units_kernel<true><<<tiles, kThreads, 0, st>>>(a);
    else
        recover_units_kernel<false><<<tiles, kThreads, 0, st>>>(a);
}

}  // namespace dev
}  // namespace xnyz
