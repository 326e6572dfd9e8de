// Compress-side stream kernels over the sorted keys.
//
//   units_*       one pass over the sorted keys: RLE run heads (unique cells), block heads,
//                 quad / repos deltas (block mode) or SFC deltas (direct mode), PFor symbols
//                 and patches, symbol histograms with first-occurrence units, all placed by
//                 a three-channel chained scan (units, patches, blocks).
//   count_stats   -rle count per unit and its histogram.
//   block_max, block_pack  BitPacker<uint64_t> of the block-id and block-count deltas.
//   encode        the entropy coders: GolombRiceCoder<uint64_t>::pack of the patches,
//                 HuffmanEncoder<T>::encode / exp-Golomb encode with host-built codes.
//   gather        the container's pieces, at any alignment; fill: the call's zeroed state.
//
// Reference (paths relative to its source/): quantizer/block_quantizer.hpp:117-149 (LCP
// streams), composer/block_compressor.hpp:110-114,146-147 (deltas), encoder/
// p_for_delta_encoder.hpp:27-43 (PFor, limit 254), encoder/golomb_rice_encoder.hpp:92-148,
// encoder/bitpacking_encoder.hpp:17-51, encoder/huffman_encoder.hpp:150-170,365-396,
// composer/block_compressor_rle.hpp:97-123,290-308 (dedup and count stream).
#include "device_common.cuh"
#include "kernels.h"

namespace xnyz {
namespace dev {

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;
static_assert(kTile == kEncTile, "tile size");

__device__ __forceinline__ void block_key_fields(u64 k, const BlockKeyParams& kp, u64& id, u32& quad, u32& sfc) {
    id = (kp.defect_flag && k >= kp.defect_flag) ? (((k - kp.defect_flag) >> 21) + kp.defect_base) : (k >> 21);
    quad = (u32)(k >> 18) & 7u;
    sfc = (u32)(k & 0x3ffffu);
}

__device__ __forceinline__ u64 direct_key_sfc(u64 k, const DirectKeyParams& kp) {
    return (kp.defect_flag && k >= kp.defect_flag) ? (kp.defect_high | (k - kp.defect_flag)) : k;
}

__device__ __forceinline__ void copy_async16(void* smem, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((u32)__cvta_generic_to_shared(smem)), "l"(g) : "memory");
}

// Units from the sorted keys.  Warp w owns keys [32 ITEMS w, 32 ITEMS (w + 1)) of the tile, 32 consecutive
// ones (one per lane) per round, so that a round's outputs land in consecutive units.  The first pass
// classifies each key against the one before it and counts; the second places, tallies and writes.  What
// a key came to (repos delta, flags, quad delta) stays in one register in between.
//
// Bound by instructions, then by the chain: classified twice, with the histogram's equal symbols found
// by masks in shared memory, a key took 308 instructions and 64M keys 718 us; this 572 (3.3 TB/s).  (The
// hardware merges equal addresses of a shared increment; the first unit of a symbol is only touched when
// it gets smaller.)  Tiles of 2048 keys take 725 us for 64M: the chain.  Tiles of 1024 below kUnitSmall,
// since a tile's rounds are serial: 1013 keys 19 -> 10 us, 120k 17 -> 13 (1M, tiles of 4096: 30 -> 22).
template <bool DIRECT, int ITEMS>
__global__ void __launch_bounds__(kThreads) units_kernel(const u64* __restrict__ keys, u64 n, int rle,
                                                         BlockKeyParams bkp, DirectKeyParams dkp, UnitOutputs out,
                                                         Status* status, u32* tile_counter, u32* err) {
    constexpr int kT = kThreads * ITEMS, kW = kThreads / 32;
    __shared__ __align__(16) u64 sk[kT + 2];  // [1] the key before the tile, [2 + e] key e
    __shared__ u32 slot;
    __shared__ u32 hrep[256], frep[256], hquad[8], fquad[8];
    __shared__ u32 wtot[kW];           // units | patches << 10 | blocks << 20 of each warp
    __shared__ u64 sbase[3];
    __shared__ unsigned long long psum;

    const u32 tile = claim_tile(tile_counter, &slot);
    const u64 base = (u64)tile * kT;
    const u32 cnt = (u32)min((u64)kT, n - base);
    const int tid = threadIdx.x, w = tid >> 5;
    const u32 lane = lane_id(), lt = lanemask_lt();
#pragma unroll
    for (int i = 0; i < ITEMS / 2; ++i) {
        const u32 e = ((u32)i * kThreads + tid) * 2u;
        if (e + 1 < cnt) copy_async16(&sk[2 + e], keys + base + e);
        else if (e < cnt) sk[2 + e] = keys[base + e];
    }
    // the very first key differs from its predecessor in every bit: a head that starts a block
    if (tid == 0) sk[1] = base ? keys[base - 1] : ~keys[0];
    hrep[tid] = 0;
    frep[tid] = 0xffffffffu;
    if (tid < 8) {
        hquad[tid] = 0;
        fquad[tid] = 0xffffffffu;
    }
    if (tid == 0) psum = 0;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    const u32 e0 = (u32)w * (32u * ITEMS) + lane;
    auto sfc_delta = [&](u32 e) -> u64 {  // direct mode
        const u64 s = direct_key_sfc(sk[2 + e], dkp);
        return base + e ? s - direct_key_sfc(sk[1 + e], dkp) : s;
    };
    constexpr u32 kHead = 1u << 18, kPatch = 1u << 19, kBlock = 1u << 20;
    u32 info[ITEMS];  // repos delta (18 bits), flags, quad delta << 21; 0: no unit
    u32 sums = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const u32 e = e0 + 32u * r;
        info[r] = 0;
        if (e < cnt) {
            const u64 k = sk[2 + e], x = k ^ sk[1 + e];
            if (!rle || x || (base + e) == 0) {
                u32 f = kHead;
                if (DIRECT) {
                    if (sfc_delta(e) > 254u) f |= kPatch;
                } else {
                    const u32 lo = (u32)k, before = lo ^ (u32)x;
                    const bool block = (x >> 21) != 0, moved = (x >> 18) != 0;
                    const u32 d = moved ? lo & 0x3ffffu : lo - before;
                    const u32 quad = ((lo >> 18) & 7u) - (block ? 0u : (before >> 18) & 7u);
                    f |= d | (quad << 21) | (d > 254u ? kPatch : 0u) | (block ? kBlock : 0u);
                }
                info[r] = f;
                sums += 1u + (f & kPatch ? 1u << 10 : 0u) + (f & kBlock ? 1u << 20 : 0u);
            }
        }
    }
    sums = __reduce_add_sync(kFullMask, sums);  // (at most 512 each)
    if (lane == 0) wtot[w] = sums;
    __syncthreads();
    u32 mu = 0, mp = 0, mb = 0;  // the warp's first unit, patch and block in the tile
#pragma unroll
    for (int i = 0; i < kW; ++i) {
        const u32 t = wtot[i];
        if (i < w) {
            mu += t & 0x3ffu;
            mp += (t >> 10) & 0x3ffu;
            mb += t >> 20;
        }
    }
    if (w == kW - 1) {  // the three counts (below 2^31) in one chained scan
        const u32 tu = mu + (sums & 0x3ffu), tp = mp + ((sums >> 10) & 0x3ffu), tb = mb + (sums >> 20);
        const Pair b = chain_lookback(status, tile, Pair{(u64)tu | ((u64)tp << 32), tb}, PairAdd{}, err);
        if (lane == 0) {
            sbase[0] = b.lo & 0xffffffffull;
            sbase[1] = b.lo >> 32;
            sbase[2] = b.hi;
            if (tile == gridDim.x - 1) {
                out.counters[0] = sbase[0] + tu;
                out.counters[1] = sbase[1] + tp;
                out.counters[2] = sbase[2] + tb;
            }
        }
    }
    __syncthreads();

    const u64 ubase = sbase[0];
    u8* const rep_sym = out.rep_sym + ubase;
    u8* const quad_sym = out.quad_sym + ubase;
    u32* const unit_pos = out.unit_pos + ubase;
    u64* const rep_val = out.rep_val ? (u64*)out.rep_val + ubase : nullptr;
    u64* const patch64 = static_cast<u64*>(out.patches) + sbase[1];
    u32* const patch32 = static_cast<u32*>(out.patches) + sbase[1];
    u64* const blk_id = (u64*)out.blk_id + sbase[2];
    u32* const blk_unit = out.blk_unit + sbase[2];
    u64 mysum = 0;
    u32 q0 = 0, q1 = 0;  // units of my quad deltas 0..3 and 4..7, one byte each
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const u32 e = e0 + 32u * r, f = info[r];
        const bool head = f != 0, patch = f & kPatch, block = !DIRECT && (f & kBlock);
        const u32 hm = __ballot_sync(kFullMask, head), pm = __ballot_sync(kFullMask, patch);
        const u32 bm = DIRECT ? 0u : __ballot_sync(kFullMask, block);
        if (head) {
            const u32 u = mu + __popc(hm & lt);
            const u64 val = DIRECT ? sfc_delta(e) : (u64)(f & 0x3ffffu);
            const u32 sym = patch ? 0u : (u32)val + 1u;
            rep_sym[u] = (u8)sym;
            if (rep_val) rep_val[u] = val;
            if (rle) unit_pos[u] = (u32)(base + e);
            if (patch) {
                const u32 at = mp + __popc(pm & lt);
                if (DIRECT) patch64[at] = val;
                else patch32[at] = (u32)val;  // 18-bit codes
                mysum += val;
            }
            atomicAdd(&hrep[sym], 1u);
            if (u < *(volatile u32*)&frep[sym]) atomicMin(&frep[sym], u);
            if (!DIRECT) {
                const u32 qd = f >> 21;
                quad_sym[u] = (u8)(qd + 1u);
                const u32 one = 1u << (8u * (qd & 3u));
                if (qd < 4u) q0 += one;
                else q1 += one;
                if (u < *(volatile u32*)&fquad[qd]) atomicMin(&fquad[qd], u);
                if (block) {
                    const u32 at = mb + __popc(bm & lt);
                    u64 id;
                    u32 quad, sfc;
                    block_key_fields(sk[2 + e], bkp, id, quad, sfc);
                    blk_id[at] = id;
                    blk_unit[at] = (u32)ubase + u;
                }
            }
        }
        mu += __popc(hm);
        mp += __popc(pm);
        mb += __popc(bm);
    }
    if (!DIRECT) {
        const u32 t[4] = {__reduce_add_sync(kFullMask, q0 & 0xff00ffu), __reduce_add_sync(kFullMask, (q0 >> 8) & 0xff00ffu),
                          __reduce_add_sync(kFullMask, q1 & 0xff00ffu), __reduce_add_sync(kFullMask, (q1 >> 8) & 0xff00ffu)};
        if (lane < 8u) {  // delta v: byte v % 4 of its word, the low or high half of t
            const u32 x = lane & 4u ? (lane & 1u ? t[3] : t[2]) : (lane & 1u ? t[1] : t[0]);
            const u32 c = lane & 2u ? x >> 16 : x & 0xffffu;
            if (c) atomicAdd(&hquad[lane], c);
        }
    }
    mysum = warp_sum(mysum);
    if (lane == 0 && mysum) atomicAdd(&psum, mysum);
    __syncthreads();
    if (tid == 0 && psum) atomicAdd(&out.counters[3], psum);
    // (first units come down with the tiles, nearly in order: read before each minimum)
    auto flush = [&](unsigned long long* hist, u32* first, u32 c, u32 f) {
        atomicAdd(hist, (unsigned long long)c);
        f += (u32)ubase;
        if (f < __ldcg(first)) atomicMin(first, f);
    };
    if (hrep[tid]) flush(out.hist_rep + tid, out.first_rep + tid, hrep[tid], frep[tid]);
    if (!DIRECT && tid < 8 && hquad[tid]) flush(out.hist_quad + tid + 1, out.first_quad + tid + 1, hquad[tid], fquad[tid]);
}

// -rle: count of each unit = distance to the next unit's first point, and the counts' histogram with
// first occurrences (kept as ~unit, so that everything starts at zero).  Most counts are 1: those are
// tallied by ballots in registers, the others go through the block's histogram.  Block b of a warp's
// sequence is read two rounds at a time (293 -> 138 us for 64M units).  units and n are device values
// when units_dev is given.
__global__ void __launch_bounds__(kThreads) count_stats_kernel(const u32* __restrict__ unit_pos, u64 units,
                                                               const unsigned long long* units_dev, u64 n,
                                                               i32* __restrict__ counts, CountStats cs) {
    __shared__ u32 sh[kCountDense], sf[kCountDense];
    __shared__ u32 smax;
    if (units_dev) units = *units_dev;
    for (int i = threadIdx.x; i < kCountDense; i += kThreads) {
        sh[i] = 0;
        sf[i] = 0u;
    }
    if (threadIdx.x == 0) smax = 0;
    __syncthreads();
    const u32 lane = lane_id();
    const u64 stride = (u64)gridDim.x * kThreads * 4;
    u32 ones = 0, one_first = 0, top = 0;
    for (u64 b0 = ((u64)blockIdx.x * kThreads + (threadIdx.x & ~31u)) * 4; b0 < units; b0 += stride) {
        u32 at[4], nx[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const u64 u = b0 + 32 * r + lane;
            if (!unit_pos) {
                nx[r] = u < units ? (u32)counts[u] : 0u;
                at[r] = 0;
            } else {
                at[r] = u < units ? __ldg(unit_pos + u) : 0u;
                nx[r] = u + 1 < units ? __ldg(unit_pos + u + 1) : (u32)n;
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const u64 u = b0 + 32 * r + lane;
            const bool ok = u < units;
            const u32 c = nx[r] - at[r];
            if (ok && unit_pos) counts[u] = (i32)c;
            const u32 m1 = __ballot_sync(kFullMask, ok && c == 1u);
            if (m1) {
                ones += (u32)__popc(m1);
                if (!one_first) one_first = ~((u32)(b0 + 32 * r) + (u32)__ffs(m1) - 1u);
            }
            if (ok && c != 1u) {
                if (c < (u32)kCountDense) {
                    atomicAdd(&sh[c], 1u);
                    if (sf[c] < ~(u32)u) atomicMax(&sf[c], ~(u32)u);
                    top = max(top, c);
                } else {
                    const u32 slot = atomicAdd(cs.over_n, 1u);
                    cs.over_val[slot] = c;
                    cs.over_unit[slot] = (u32)u;
                }
            }
        }
    }
    if (lane == 0 && ones) {
        atomicAdd(&sh[1], ones);
        atomicMax(&sf[1], one_first);
        top = max(top, 1u);
    }
    if (top) atomicMax(&smax, top);
    __syncthreads();
    const u32 last = smax;
    for (u32 i = threadIdx.x; i <= last; i += kThreads)
        if (sh[i]) {
            atomicAdd(&cs.bins[i].n, (u64)sh[i]);
            atomicMax(&cs.bins[i].inv_first, sf[i]);
        }
    if (threadIdx.x == 0 && last) atomicMax(cs.max_dense, last);
}

// Block b's id delta and count delta (u64, wrapping like the reference's in-place differences).
__device__ __forceinline__ void block_deltas(const u64* __restrict__ blk_id, const u32* __restrict__ blk_unit, u64 nb,
                                             u32 units, u64 b, u64& db, u64& dc) {
    const u64 id = __ldg(blk_id + b), pid = b ? __ldg(blk_id + b - 1) : 0ull;
    const u32 un = __ldg(blk_unit + b), next = b + 1 < nb ? __ldg(blk_unit + b + 1) : units;
    db = id - pid;
    dc = next - un;
    if (b) dc -= (u64)(un - __ldg(blk_unit + b - 1));
}

// Largest id delta and count delta (the bit widths of the two block streams).  Reads 12 B per block;
// a thread takes four consecutive blocks.
__global__ void __launch_bounds__(kThreads) block_max_kernel(const u64* __restrict__ blk_id,
                                                             const u32* __restrict__ blk_unit,
                                                             const unsigned long long* __restrict__ counters, u64* max2) {
    const u64 nb = counters[2];
    const u32 units = (u32)counters[0];
    __shared__ u64 sm[2][kThreads / 32];
    u64 m0 = 0, m1 = 0;
    const u64 stride = (u64)gridDim.x * kThreads * 4;
    for (u64 b = ((u64)blockIdx.x * kThreads + threadIdx.x) * 4; b < nb; b += stride) {
        if (b + 4 < nb) {  // (arrays start on 256-byte boundaries)
            const ulonglong2 i0 = __ldg(reinterpret_cast<const ulonglong2*>(blk_id + b)),
                             i1 = __ldg(reinterpret_cast<const ulonglong2*>(blk_id + b + 2));
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(blk_unit + b));
            const u32 u4 = __ldg(blk_unit + b + 4);
            const u64 pid = b ? __ldg(blk_id + b - 1) : 0ull;
            const u32 pu = b ? __ldg(blk_unit + b - 1) : 0u;
            m0 = max(max(m0, i0.x - pid), max(i0.y - i0.x, max(i1.x - i0.y, i1.y - i1.x)));
            const u64 c = u.x - pu, c0 = u.y - u.x, c1 = u.z - u.y, c2 = u.w - u.z, c3 = u4 - u.w;
            m1 = max(max(m1, b ? c0 - c : c0), max(c1 - c0, max(c2 - c1, c3 - c2)));
        } else {
            for (u64 x = b; x < nb; ++x) {
                u64 db, dc;
                block_deltas(blk_id, blk_unit, nb, units, x, db, dc);
                m0 = max(m0, db);
                m1 = max(m1, dc);
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        m0 = max(m0, __shfl_xor_sync(kFullMask, m0, d));
        m1 = max(m1, __shfl_xor_sync(kFullMask, m1, d));
    }
    if (lane_id() == 0) {
        sm[0][threadIdx.x >> 5] = m0;
        sm[1][threadIdx.x >> 5] = m1;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        u64 m = 0;
        for (int w = 0; w < kThreads / 32; ++w) m = max(m, sm[threadIdx.x][w]);
        if (m) atomicMax(&max2[threadIdx.x], m);
    }
}

// One block stream on its way out: BitPacker (value b at bit b * width, LSB-first) into bytes
// [dst, dst + len), dst at any byte (widths 8..64), or OR-ed into the zeroed words at `words`.
struct PackStream {
    u8* dst;
    u64 len;
    u32* words;
    int width;
    u32 magic;  // ceil(2^32 / width): x / width for x width < 2^32
};

constexpr int kPackTile = 2048;  // blocks per thread block; their bits fill 64 `width` whole words
constexpr int kPackHead = 4;     // values before the tile (at most 24 bits of them reach into its first word)
constexpr int kPackTail = 5;     // zeros after the last value, for the last word

// The tile's bits of one stream from its values v[0 .. kPackHead + kPackTile) in shared memory (the
// first kPackHead precede the tile, kPackTail follow it).  Thread-per-word: aligned word i of dst holds
// stream bits [32 i - 8 m, 32 i - 8 m + 32) past the tile's first, m the bytes dst lies past a
// 4-byte boundary, from the one or two (widths below 32: up to five) values that overlap them.
__device__ __forceinline__ void pack_tile(const PackStream& s, const u64* v, u64 tile, u64 nb) {
    const u32 wu = (u32)s.width;
    if (wu < (u32)kPackDirectWidth) {
        for (u32 i = threadIdx.x & ~31u; i < (u32)kPackTile; i += kThreads) {
            const u64 b = tile * kPackTile + i + lane_id();
            warp_write_lsb(s.words, b * wu, v[kPackHead + i + lane_id()], b < nb ? wu : 0u);
        }
        return;
    }
    const u32 m = (u32)(reinterpret_cast<uintptr_t>(s.dst) & 3u);
    const u64 w0 = tile * 64 * wu;
    u32* const out = reinterpret_cast<u32*>(s.dst - m) + w0;
    const u32 left = (u32)min(nb - tile * kPackTile, (u64)kPackTile);
    const u32 nwords = (left * wu + 8 * m + 31) / 32;  // the last tile's end with the stream
    const u32 mine = left == (u32)kPackTile && (tile + 1) * kPackTile < nb ? 64 * wu : nwords;
    const i64 first = 4 * (i64)w0 - (i64)m;  // stream byte of word 0
    for (u32 i = threadIdx.x; i < mine; i += kThreads) {
        const u32 q = 32 * i + kPackHead * wu - 8 * m;
        u32 x = __umulhi(q, s.magic);
        const u32 r = q - x * wu;
        u32 word = (u32)(v[x] >> r), got = wu - r;
        while (got < 32u) {
            word |= (u32)v[++x] << got;
            got += wu;
        }
        const i64 at = first + 4 * (i64)i;
        if (at >= 0 && at + 4 <= (i64)s.len) {
            out[i] = word;
        } else {
            for (int b = 0; b < 4; ++b)
                if (at + b >= 0 && at + b < (i64)s.len) reinterpret_cast<u8*>(out + i)[b] = (u8)(word >> (8 * b));
        }
    }
}

// Both block streams from the block ids and first units: 12 B read and the packed bits written per
// block, straight to where the container has them; what bounds it is the instructions per word.  For
// the 64M blocks of 64M terrain points at L2 0.001 (42 and 64 bits): deltas through memory, a
// bit-pack pass each with shuffles and a copy into the container took 394 + 860 + 600 us, shuffles
// alone from the ids 1044, words from shared memory (this kernel) 442 and
// block_max 132.
__global__ void __launch_bounds__(kThreads) block_pack_kernel(const u64* __restrict__ blk_id,
                                                              const u32* __restrict__ blk_unit, u64 nb, u32 units,
                                                              PackStream s0, PackStream s1) {
    __shared__ u64 v0[kPackHead + kPackTile + kPackTail], v1[kPackHead + kPackTile + kPackTail];
    const u64 tile = blockIdx.x;
    const u64 mask0 = s0.width >= 64 ? ~0ull : ((1ull << s0.width) - 1), mask1 = s1.width >= 64 ? ~0ull : ((1ull << s1.width) - 1);
    for (int i = threadIdx.x; i < kPackHead + kPackTile + kPackTail; i += kThreads) {
        const i64 b = (i64)(tile * kPackTile) + i - kPackHead;
        u64 db = 0, dc = 0;
        if (b >= 0 && b < (i64)nb) block_deltas(blk_id, blk_unit, nb, units, (u64)b, db, dc);
        v0[i] = db & mask0;
        v1[i] = dc & mask1;
    }
    __syncthreads();
    pack_tile(s0, v0, tile, nb);
    pack_tile(s1, v1, tile, nb);
}

// ---------------------------------------------------------------- entropy coders ---------
// A container's entropy coders (Golomb-Rice patches, repos / SFC symbols, quad symbols, counts) are
// independent and run in one launch: each takes a range of the blocks.  (Four launches on side
// streams forked and joined by events cost 13 more calls.)  Within a coder, tiles of 4096 values
// are chained by their code lengths; fixed-length codes need no chain.
constexpr u32 kStageWords = 5632;  // a tile's output: 44 bits per value
union EncodeShared {
    struct {
        u64 scratch[16];
        u64 sbase;
        u32 slot;
        u64 table[256];  // byte symbols: length << 32 | code
        u32 out[kStageWords];
    } c;
    u32 fixed[256];
};

__device__ __forceinline__ u64 tile_bit_base(const EncodeJob& j, u32 tile, u64 tot, u64* sbase, u32* err) {
    if (threadIdx.x < 32) {
        const u64 before = chain_add(j.status, tile, tot, err);
        if (threadIdx.x == 0) {
            *sbase = before;
            if (tile == j.blocks - 1) *j.total_bits = before + tot;
        }
    }
    __syncthreads();
    return *sbase;
}

// Where a tile's codewords (tot bits from stream bit `base`) are assembled: in shared memory, zeroed
// here, when they fit, and then stored as whole words (the first and the last, shared with the
// neighbouring tiles, are OR-ed); else straight in the output.  A thread's words lie some ten words
// from the next thread's, so stores from the threads' runs touch a sector each: from shared memory
// 64M Golomb-Rice codes of 18.5 bits take 388 us (464 with a look-back over 32 tiles a step, straight
// and so 492).
struct TileWriter {
    u32* words;
    u64 first;  // output word that `words` starts with
    bool staged;
    __device__ __forceinline__ TileWriter(const EncodeJob& j, EncodeShared& sh, u64 base, u64 tot) {
        first = base >> 5;
        const u64 n = ((base & 31u) + tot + 31) >> 5;
        staged = n <= kStageWords;
        words = staged ? sh.c.out : j.words + first;
        if (staged)
            for (u32 i = threadIdx.x; i < (u32)n; i += kThreads) sh.c.out[i] = 0u;
        __syncthreads();
    }
    __device__ __forceinline__ void finish(const EncodeJob& j, const EncodeShared& sh, u64 base, u64 tot) const {
        if (!staged) return;
        __syncthreads();
        const u32 n = (u32)(((base & 31u) + tot + 31) >> 5);
        for (u32 i = threadIdx.x; i < n; i += kThreads) {
            const u32 v = sh.c.out[i];
            if (i == 0 || i + 1 == n) {
                if (v) atomicOr(&j.words[first + i], v);
            } else {
                j.words[first + i] = v;
            }
        }
    }
};

// Sixteen consecutive values of a thread, whole 16-byte loads where they are all there.
template <typename T>
__device__ __forceinline__ void load16(const T* __restrict__ in, u32 have, T (&v)[16]) {
    if (have >= 16u) {
        constexpr int kVec = 16 / sizeof(T);
#pragma unroll
        for (int i = 0; i < 16; i += kVec) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(in + i));
            const u32 w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < kVec; ++e) {
                if (sizeof(T) == 8) v[i + e] = (T)((u64)w[2 * e] | ((u64)w[2 * e + 1] << 32));
                else if (sizeof(T) == 4) v[i + e] = (T)w[e];
                else v[i + e] = (T)(w[e / 4] >> (8 * (e % 4)));
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = i < (int)have ? in[i] : (T)0;
    }
}

// Thread t codes the tile's values [16 t, 16 t + 16) as one run of consecutive codewords, kept in
// registers for the length sum and the writes; the run's bits leave a word at a time (LsbRun).
template <typename T>
__device__ __forceinline__ void gr_encode_tile(const EncodeJob& j, EncodeShared& sh, u32* err) {
    const int k = j.k;
    const u32 tile = claim_tile(j.tile_counter, &sh.c.slot);
    const u64 base = (u64)tile * kTile;
    const u32 cnt = (u32)min((u64)kTile, j.n - base);
    const u32 e0 = threadIdx.x * kItems;
    const u32 have = e0 < cnt ? min(cnt - e0, 16u) : 0u;
    T v[16];
    load16(static_cast<const T*>(j.in) + base + e0, have, v);
    u64 sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i)
        if (i < (int)have) sum += ((u64)v[i] >> k) + 1u + (u64)k;
    u64 tot;
    const u64 ex = block_exclusive<kThreads>(sum, 0ull, AddOp{}, sh.c.scratch, tot);
    const u64 at = tile_bit_base(j, tile, tot, &sh.c.sbase, err);
    if (at + tot > j.cap_bits) {  // output bound (never reached with valid sizes)
        if (tot) atomicOr(err, kErrOverflow);
        return;
    }
    const TileWriter out(j, sh, at, tot);
    const u64 pos = (at & 31u) + ex;
    const u64 mask = k ? ((1ull << k) - 1) : 0ull;
    LsbRun run;
    run.begin(out.words, pos);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (i >= (int)have) continue;
        const u64 q = (u64)v[i] >> k;
        const u64 r = (u64)v[i] & mask;
        if (q + 1u + (u64)k <= 32u) {  // unary part, terminating zero and remainder in one piece
            run.put32((u32)((q ? ((1ull << q) - 1) : 0ull) | (r << (q + 1))), (u32)(q + 1u + (u64)k));
        } else {
            run.ones(q);
            run.put32(0u, 1u);
            run.put(r, (u32)k);
        }
    }
    run.end();
    out.finish(j, sh, at, tot);
}

__device__ __forceinline__ void huff_encode_tile(const EncodeJob& j, EncodeShared& sh, u32* err) {
    const ByteCodes* codes = static_cast<const ByteCodes*>(j.codes);
    sh.c.table[threadIdx.x] = ((u64)codes->len[threadIdx.x] << 32) | codes->bits[threadIdx.x];
    const u32 tile = claim_tile(j.tile_counter, &sh.c.slot);
    const u64 base = (u64)tile * kTile;
    const u32 cnt = (u32)min((u64)kTile, j.n - base);
    const u32 e0 = threadIdx.x * kItems;
    const u32 have = e0 < cnt ? min(cnt - e0, 16u) : 0u;
    u8 v[16];
    load16(static_cast<const u8*>(j.in) + base + e0, have, v);
    u64 sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i)
        if (i < (int)have) sum += sh.c.table[v[i]] >> 32;
    u64 tot;
    const u64 ex = block_exclusive<kThreads>(sum, 0ull, AddOp{}, sh.c.scratch, tot);
    const u64 at = tile_bit_base(j, tile, tot, &sh.c.sbase, err);
    if (at + tot > j.cap_bits) {  // output bound (never reached with valid sizes)
        if (tot) atomicOr(err, kErrOverflow);
        return;
    }
    const TileWriter out(j, sh, at, tot);
    const u64 pos = (at & 31u) + ex;
    MsbRun run;
    run.begin(out.words, pos);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (i >= (int)have) continue;
        const u64 e = sh.c.table[v[i]];
        const u32 len = (u32)(e >> 32);
        // Codes longer than 32 bits are the 32-bit value zero-extended (huffman_encoder.hpp:251).
        if (len > 32u) {
            run.zeros(len - 32u);
            run.put32((u32)e, 32u);
        } else {
            run.put32((u32)e, len);
        }
    }
    run.end();
    out.finish(j, sh, at, tot);
}

// A prefix code whose codewords all have one length L (1..24 bits): symbol i occupies stream
// bits [i L, (i + 1) L), so no scan is needed.  Thread g codes symbols [32 g, 32 g + 32), whose
// 32 L bits fill exactly words [g L, g L + L), MSB-first and stored byte-swapped as MsbRun
// stores them; whole words, no atomics.  Symbols index j.bits (counts: the dense table).
template <typename T>
__device__ __forceinline__ void fixed_encode_block(const EncodeJob& j, EncodeShared& sh, u32 block) {
    const int len = j.k;
    sh.fixed[threadIdx.x] = __ldg(&j.bits[threadIdx.x]);
    __syncthreads();
    const u64 g = (u64)block * kThreads + threadIdx.x;
    const u64 total = j.n * (u64)len;
    if (g == 0) *j.total_bits = total;
    const u64 s0 = g * 32u;
    if (s0 >= j.n) return;
    const u32 mask = (1u << len) - 1u;
    u64 acc = 0, w = g * (u64)len;
    u32 nb = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const u64 s = s0 + 16u * h;
        const u32 have = s < j.n ? (u32)min(j.n - s, (u64)16) : 0u;
        T v[16];
        load16(static_cast<const T*>(j.in) + s, have, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const u32 x = (u32)v[i];
            const u32 c = i < (int)have ? ((sizeof(T) == 1 || x < 256u ? sh.fixed[x & 255u] : __ldg(&j.bits[x])) & mask) : 0u;
            acc = (acc << len) | c;
            nb += (u32)len;
            if (nb >= 32u) {
                nb -= 32u;
                if (w * 32u < total) j.words[w] = __byte_perm((u32)(acc >> nb), 0, 0x0123);
                ++w;
            }
        }
    }
}

__device__ __forceinline__ u32 rev_low(u64 v, int k) { return k ? (__brev((u32)v) >> (32 - k)) : 0u; }

__device__ __forceinline__ void count_encode_tile(const EncodeJob& j, EncodeShared& sh, u32* err) {
    const u32 tile = claim_tile(j.tile_counter, &sh.c.slot);
    const u64 base = (u64)tile * kTile;
    const u32 cnt = (u32)min((u64)kTile, j.n - base);
    const u32 e0 = threadIdx.x * kItems;
    const u32 have = e0 < cnt ? min(cnt - e0, 16u) : 0u;
    i32 v[16];
    load16(static_cast<const i32*>(j.in) + base + e0, have, v);
    const int eg_k = j.k;
    // code of one count: (length, value bits, bit offset of the value inside the code)
    auto code = [&](i32 c, u32& len, u64& val, u32& nb) {
        if (eg_k >= 0) {
            const long long s = c;
            const u64 z = ((u64)s << 1) ^ (u64)(s >> 63);
            const u64 n1 = (z >> eg_k) + 1u;
            const u32 lz = bitlen64(n1) - 1u;
            len = 2u * lz + 1u + (u32)eg_k;
            nb = lz + 1u + (u32)eg_k;
            val = (n1 << eg_k) | rev_low(z, eg_k);
        } else {
            const u32 uc = (u32)c;
            u32 bits = 0, l = 0;
            if (uc < (u32)kCountDense) {
                bits = __ldg(&j.bits[uc]);
                l = __ldg(&j.len[uc]);
            } else {
                u32 lo = 0, hi = j.sparse_n;
                while (lo < hi) {
                    const u32 mid = (lo + hi) >> 1;
                    if (j.sparse_val[mid] < uc) lo = mid + 1; else hi = mid;
                }
                if (lo < j.sparse_n && j.sparse_val[lo] == uc) {
                    bits = j.sparse_bits[lo];
                    l = j.sparse_len[lo];
                } else {
                    atomicOr(err, kErrOverflow);
                }
            }
            len = l;
            nb = l > 32u ? 32u : l;
            val = bits;
        }
    };
    u64 sum = 0;
#pragma unroll 4
    for (int i = 0; i < kItems; ++i)
        if (i < (int)have) {
            u32 len, nb;
            u64 val;
            code(v[i], len, val, nb);
            sum += len;
        }
    u64 tot;
    const u64 ex = block_exclusive<kThreads>(sum, 0ull, AddOp{}, sh.c.scratch, tot);
    const u64 at = tile_bit_base(j, tile, tot, &sh.c.sbase, err);
    if (at + tot > j.cap_bits) {  // output bound (never reached with valid sizes)
        if (tot) atomicOr(err, kErrOverflow);
        return;
    }
    const TileWriter out(j, sh, at, tot);
    const u64 pos = (at & 31u) + ex;
    MsbRun run;
    run.begin(out.words, pos);
#pragma unroll 4
    for (int i = 0; i < kItems; ++i) {
        if (i >= (int)have) continue;
        u32 len, nb;
        u64 val;
        code(v[i], len, val, nb);
        run.zeros(len - nb);  // exp-Golomb's leading zeros, or a long Huffman code's extension
        run.put(val, nb);
    }
    run.end();
    out.finish(j, sh, at, tot);
}

__global__ void __launch_bounds__(kThreads) encode_kernel(const __grid_constant__ EncodeArgs a) {
    __shared__ EncodeShared sh;
    u32 b = blockIdx.x;
    int i = 0;
    while (b >= a.job[i].blocks) b -= a.job[i++].blocks;
    const EncodeJob& j = a.job[i];
    switch (j.kind) {
        case kEncodeGolombRice32: gr_encode_tile<u32>(j, sh, a.err); break;
        case kEncodeGolombRice64: gr_encode_tile<u64>(j, sh, a.err); break;
        case kEncodeHuffman: huff_encode_tile(j, sh, a.err); break;
        case kEncodeFixedU8: fixed_encode_block<u8>(j, sh, b); break;
        case kEncodeFixedI32: fixed_encode_block<i32>(j, sh, b); break;
        default: count_encode_tile(j, sh, a.err); break;
    }
}

// Sets ranges of 4-byte words (a call's counters, histograms, look-back flags and OR-ed output words)
// in one launch instead of a memset each.
__global__ void __launch_bounds__(kThreads) fill_kernel(const __grid_constant__ FillArgs a) {
    const u64 t = (u64)blockIdx.x * kThreads + threadIdx.x, stride = (u64)gridDim.x * kThreads;
    for (int i = 0; i < a.count; ++i) {
        const FillRange r = a.range[i];
        u32* p = static_cast<u32*>(r.p);
        const u64 head = min((u64)r.words, (u64)((16u - (u32)(reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) / 4u);
        const u64 vecs = (r.words - head) / 4;
        uint4* v = reinterpret_cast<uint4*>(p + head);
        for (u64 x = t; x < vecs; x += stride) v[x] = make_uint4(r.value, r.value, r.value, r.value);
        if (t < head) p[t] = r.value;
        if (t < r.words - head - 4 * vecs) p[head + 4 * vecs + t] = r.value;
    }
}

// One block per 16 KB of the destination (by its address) and piece.  The body goes out 16 bytes per
// store, the source read as aligned words and shifted to the destination's alignment; the bytes
// before and after it one by one.
constexpr u64 kGatherChunk = 16384;
__global__ void __launch_bounds__(kThreads) gather_kernel(const __grid_constant__ GatherArgs a, u8* __restrict__ dst) {
    u64 c = blockIdx.x;
    const u64 late = a.late_bits ? min((u64)(*a.late_bits + 7) / 8, (u64)a.late_most) : 0ull;
    for (int i = 0; i < a.count; ++i) {
        const GatherPiece& p = a.piece[i];
        const u64 len = p.kind == kGatherLate ? late : p.len;
        const u64 d0 = reinterpret_cast<u64>(dst) + p.off + (p.after ? late : 0ull), d1 = d0 + len;
        const u64 chunks = len ? (d1 - 1) / kGatherChunk - d0 / kGatherChunk + 1 : 0ull;
        if (c >= chunks) {
            c -= chunks;
            continue;
        }
        const u64 base = (d0 / kGatherChunk + c) * kGatherChunk;
        const u64 lo = max(base, d0), hi = min(base + kGatherChunk, d1);
        if (!p.src) {
            for (u64 x = lo + threadIdx.x; x < hi; x += kThreads)
                *reinterpret_cast<u8*>(x) = p.kind == kGatherZero      ? (u8)0
                                            : p.kind == kGatherLateLen ? (u8)(late >> (8 * (x - d0)))
                                                                       : a.inline_bytes[p.inline_off + (u32)(x - d0)];
            return;
        }
        const u64 s0 = reinterpret_cast<u64>(p.src) - d0;  // source address = destination address + s0
        const u64 b0 = min((lo + 15) & ~15ull, hi), b1 = max(hi & ~15ull, b0);
        for (u64 x = b0 + 16 * threadIdx.x; x < b1; x += 16 * kThreads) {
            const u64 s = x + s0;
            const u32* w = reinterpret_cast<const u32*>(s & ~3ull);
            const u32 sh = (u32)(s & 3u) * 8u;
            const u32 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3), w4 = sh ? __ldg(w + 4) : 0u;
            *reinterpret_cast<uint4*>(x) = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                                                      __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
        }
        const u32 head = (u32)(b0 - lo), tail = (u32)(hi - b1);
        if (threadIdx.x < head) {
            *reinterpret_cast<u8*>(lo + threadIdx.x) = *reinterpret_cast<const u8*>(lo + threadIdx.x + s0);
        } else if (threadIdx.x >= 32u && threadIdx.x - 32u < tail) {
            const u64 x = b1 + threadIdx.x - 32u;
            *reinterpret_cast<u8*>(x) = *reinterpret_cast<const u8*>(x + s0);
        }
        return;
    }
}

inline int persistent_grid(u64 n) {
    u64 want = (n + kThreads - 1) / kThreads;
    if (want < 1) want = 1;
    return (int)(want < 148ull * 8ull ? want : 148ull * 8ull);
}

}  // namespace

template <bool DIRECT>
static void launch_units(const unsigned long long* keys, uint64_t n, int rle, const BlockKeyParams& bkp,
                         const DirectKeyParams& dkp, UnitOutputs out, ScanStatus status, uint32_t* tile_counter,
                         uint32_t* err, cudaStream_t st) {
    const unsigned tiles = (unsigned)((n + unit_tile(n) - 1) / unit_tile(n));
    if (!tiles) return;
    auto k = unit_tile(n) == kUnitTile ? units_kernel<DIRECT, kUnitTile / kThreads> : units_kernel<DIRECT, kUnitTileSmall / kThreads>;
    k<<<tiles, kThreads, 0, st>>>(reinterpret_cast<const u64*>(keys), n, rle, bkp, dkp, out, static_cast<Status*>(status),
                                  tile_counter, err);
}
void launch_units_block(const unsigned long long* keys, uint64_t n, int rle, BlockKeyParams kp, UnitOutputs out,
                        ScanStatus status, uint32_t* tile_counter, uint32_t* err, cudaStream_t st) {
    launch_units<false>(keys, n, rle, kp, DirectKeyParams{}, out, status, tile_counter, err, st);
}
void launch_units_direct(const unsigned long long* keys, uint64_t n, int rle, DirectKeyParams kp, UnitOutputs out,
                         ScanStatus status, uint32_t* tile_counter, uint32_t* err, cudaStream_t st) {
    launch_units<true>(keys, n, rle, BlockKeyParams{}, kp, out, status, tile_counter, err, st);
}
void launch_count_stats(const uint32_t* unit_pos, uint64_t units, const unsigned long long* units_dev, uint64_t n,
                        int32_t* counts, CountStats cs, cudaStream_t st) {
    count_stats_kernel<<<persistent_grid((units + 3) / 4), kThreads, 0, st>>>(unit_pos, units, units_dev, n, counts, cs);
}
void launch_block_max(const unsigned long long* blk_id, const uint32_t* blk_unit, uint64_t most_blocks,
                      const unsigned long long* counters, unsigned long long* max2, cudaStream_t st) {
    block_max_kernel<<<persistent_grid((most_blocks + 3) / 4), kThreads, 0, st>>>(blk_id, blk_unit, counters, max2);
}
void launch_block_pack(const unsigned long long* blk_id, const uint32_t* blk_unit, uint64_t nblocks, uint64_t units,
                       const BlockPackDst& blk, const BlockPackDst& cnt, cudaStream_t st) {
    if (!nblocks) return;
    auto stream = [&](const BlockPackDst& d) {
        PackStream s{};
        s.dst = d.dst;
        s.len = (nblocks * (u64)d.width + 7) / 8;
        s.words = d.words;
        s.width = d.width;
        s.magic = (u32)(((1ull << 32) + d.width - 1) / d.width);  // (width 1: not used)
        return s;
    };
    const unsigned blocks = (unsigned)((nblocks + kPackTile - 1) / kPackTile);
    block_pack_kernel<<<blocks, kThreads, 0, st>>>(blk_id, blk_unit, nblocks, (u32)units, stream(blk), stream(cnt));
}
void launch_fill(const FillArgs& a, cudaStream_t st) {
    u64 most = 0;
    for (int i = 0; i < a.count; ++i) most = a.range[i].words > most ? a.range[i].words : most;
    if (most) fill_kernel<<<persistent_grid((most + 3) / 4), kThreads, 0, st>>>(a);
}
void launch_gather(const GatherArgs& a, uint8_t* dst, cudaStream_t st) {
    u64 blocks = 0;
    for (int i = 0; i < a.count; ++i) {
        // at most this many, wherever the late stream's length puts the piece
        if (a.piece[i].len) blocks += (a.piece[i].len + kGatherChunk - 2) / kGatherChunk + 1;
    }
    if (blocks) gather_kernel<<<(unsigned)blocks, kThreads, 0, st>>>(a, dst);
}
void launch_encode(EncodeArgs a, cudaStream_t st) {
    u64 blocks = 0;
    for (int i = 0; i < a.count; ++i) {
        const u64 per = a.job[i].kind == kEncodeFixedU8 || a.job[i].kind == kEncodeFixedI32 ? 32ull * kThreads : (u64)kTile;
        a.job[i].blocks = (u32)((a.job[i].n + per - 1) / per);
        blocks += a.job[i].blocks;
    }
    if (blocks) encode_kernel<<<(unsigned)blocks, kThreads, 0, st>>>(a);
}

}  // namespace dev
}  // namespace xnyz
