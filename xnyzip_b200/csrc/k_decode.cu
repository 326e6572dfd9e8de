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
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;
static_assert(kTile == kScanTile, "tile size");

// x / d for an invariant divisor (U64Div, kernels.h)
__device__ __forceinline__ u64 udiv(u64 x, const U64Div& d) {
    const u64 t = __umul64hi(d.m, x);
    return (t + ((x - t) >> d.sh1)) >> d.sh2;
}

// ------------------------------------------------------------- block streams -----------
// The -normal/-rle block streams of block mode in one pass (block_decompressor.hpp:111-161):
// bit-unpack the block-id deltas and block-count deltas, inclusive prefix sums of both
// (u64, wrapping), the exclusive prefix of the counts (first unit of each block), and the
// per-unit block-start marks of recover_from_lcp_meta (block_quantizer.hpp:167-176).
// Within a tile the count channel carries (sum of deltas, blocks, sum of counts):
//   (A1, N1, B1) then (A2, N2, B2) = (A1 + A2, N1 + N2, B1 + B2 + N2 * A1);
// across tiles one chained scan gives the tile's true first count, and so its true sum of counts,
// which the next one chains.
struct Tri {
    u64 a, n, b;
};
struct TriOp {
    __device__ __forceinline__ Tri operator()(Tri x, Tri y) const { return Tri{x.a + y.a, x.n + y.n, x.b + y.b + y.n * x.a}; }
};

__global__ void __launch_bounds__(kThreads) block_streams_kernel(const u32* __restrict__ wb, u64 bb, int width_b,
                                                                 const u32* __restrict__ wc, u64 bc, int width_c,
                                                                 u64 nb, u64 units, u64* __restrict__ blk_out,
                                                                 u8* __restrict__ is_start, u32* __restrict__ start_block,
                                                                 ScanStatus status, u32* tile_counter,
                                                                 unsigned long long* count_total, u32* err) {
    constexpr int kWarps = kThreads / 32;
    __shared__ u32 slot;
    __shared__ u64 wsb[kWarps + 1];
    __shared__ Tri wtc[kWarps + 1];
    __shared__ u64 base_b;
    __shared__ Tri base_c;
    const u32 tile = claim_tile(tile_counter, &slot);
    const u32 ntiles = gridDim.x;
    const int tid = threadIdx.x;
    const int w = tid >> 5;
    const u32 lane = lane_id();
    // warp w owns blocks [512 w, 512 w + 512) of the tile, 32 consecutive blocks per round
    const u64 wfirst = (u64)tile * kTile + (u64)w * (32u * kItems);
    const u64 mb = width_b >= 64 ? ~0ull : ((1ull << width_b) - 1), mc = width_c >= 64 ? ~0ull : ((1ull << width_c) - 1);
    auto delta_b = [&](u64 j) { return width_b ? (peek_lsb64(wb, bb + j * (u64)width_b) & mb) : 0ull; };
    auto delta_c = [&](u64 j) { return width_c ? (peek_lsb64(wc, bc + j * (u64)width_c) & mc) : 0ull; };

    // Running values along the warp's blocks: blk (block id), cnt (block count = inclusive
    // sum of the count deltas), start (first unit of the block = exclusive sum of the
    // counts).  The warp's aggregates need no scans (below); the pass from the true carries
    // writes the outputs.
    auto pass = [&](u64& blk, u64& cnt, u64& start) {
        for (int r = 0; r < kItems; ++r) {
            const u64 j = wfirst + (u64)r * 32u + lane;
            const bool valid = j < nb;
            const u64 db = valid ? delta_b(j) : 0ull, dc = valid ? delta_c(j) : 0ull;
            const u64 bj = blk + warp_incl_add(db);
            const u64 cj = cnt + warp_incl_add(dc);
            const u64 vc = valid ? cj : 0ull;
            const u64 ci = warp_incl_add(vc);
            const u64 sj = start + ci - vc;
            blk = __shfl_sync(kFullMask, bj, 31);
            cnt = __shfl_sync(kFullMask, cj, 31);
            start += __shfl_sync(kFullMask, ci, 31);
            if (valid) {
                blk_out[j] = bj;
                if (cj > 0 && sj < units) {  // non-empty block (the reference skips empty ones)
                    is_start[sj] = 1;
                    start_block[sj] = (u32)j;
                }
            }
        }
    };
    {
        // From zero carries the warp ends at blk = sum of db, cnt = sum of dc, and start = the
        // sum of its m blocks' counts c_j = dc_0 + .. + dc_j, which is the sum over i of
        // dc_i * (m - i) (u64, wrapping like the running sums).
        const u64 wbeg = wfirst < nb ? wfirst : nb;
        const u64 nvalid = (nb - wbeg) < 32u * kItems ? nb - wbeg : 32u * kItems;
        u64 sb = 0, sc = 0, sw = 0;
        for (int r = 0; r < kItems; ++r) {
            const u64 i = (u64)r * 32u + lane;
            if (wfirst + i < nb) {
                const u64 dc = delta_c(wfirst + i);
                sb += delta_b(wfirst + i);
                sc += dc;
                sw += dc * (nvalid - i);
            }
        }
        sb = warp_sum(sb);
        sc = warp_sum(sc);
        sw = warp_sum(sw);
        if (lane == 0) {
            wsb[w] = sb;
            wtc[w] = Tri{sc, nvalid, sw};
        }
    }
    __syncthreads();
    if (tid == 0) {
        warps_exclusive<kWarps>(wsb, 0ull, AddOp{});
        warps_exclusive<kWarps>(wtc, Tri{0, 0, 0}, TriOp{});
    }
    __syncthreads();
    if (tid < 32) {
        const u64 r = chain_add(status, tile, wsb[kWarps], err);
        if (tid == 0) base_b = r;
    } else if (tid < 64) {
        Status* st = static_cast<Status*>(status) + ntiles;
        const Tri mine = wtc[kWarps];
        const u64 cnt0 = chain_add(st, tile, mine.a, err);
        const u64 sum = mine.b + mine.n * cnt0;
        const u64 first = chain_add(st + ntiles, tile, sum, err);
        if (tid == 32) {
            base_c = Tri{cnt0, 0, first};
            if (tile == ntiles - 1) *count_total = first + sum;
        }
    }
    __syncthreads();
    const Tri pre = TriOp{}(base_c, wtc[w]);
    u64 blk = base_b + wsb[w], cnt = pre.a, start = pre.b;
    pass(blk, cnt, start);
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

__global__ void __launch_bounds__(kThreads) count_total_kernel(const i32* __restrict__ c, u64 n,
                                                               unsigned long long* total) {
    u64 s = 0;
    for (u64 i = (u64)blockIdx.x * kThreads + threadIdx.x; i < n; i += (u64)gridDim.x * kThreads)
        s += (u64)max(c[i], 0);
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(kFullMask, s, d);
    if (lane_id() == 0 && s) atomicAdd(total, s);
}

// ------------------------------------------------------------- recover units -------------
struct RecoverArgs {
    const u8* rep_sym;
    const void* rep_patch;
    int patch32;
    u64 npatch;
    const u8* quad_sym;
    const u8* is_start;
    const u32* start_block;
    const u64* blk_ids;
    u64 nblocks;
    const i32* counts;
    const u64* rep_val;
    u64 units;
    u64 nout;
    RecoverParams rp;
    const u8* hinv;
    Status* status;  // [3][ntiles]: zero symbols; counts; segments (block mode) or SFC sums
    u32* tile_counter;
    float* out;
    u32* err;
};

// Block mode's segmented sums in one chained scan.  lo: repos sum since the last repos head; hi: block
// index (bits 0..31) and quad sum modulo 8 (32..34) since the last block start, whether a block starts
// (35) and whether a repos head is inside (36).
struct SegPair {
    __device__ __forceinline__ Pair operator()(Pair a, Pair b) const {
        const bool hq = (b.hi >> 35) & 1u, hr = (b.hi >> 36) & 1u;
        const u64 quad = ((hq ? 0ull : a.hi >> 32) + (b.hi >> 32)) & 7u;
        const u64 blk = ((hq ? 0ull : a.hi) + b.hi) & 0xffffffffull;
        return Pair{(hr ? 0ull : a.lo) + b.lo, blk | (quad << 32) | ((a.hi | b.hi) & (3ull << 35))};
    }
};

// Quad index step of a packed quad symbol (see recover_units_kernel): q - 1 modulo 8, 0 for
// the patch symbol 0.
__device__ __forceinline__ u32 quad_step(u32 sq) { return (sq & 8u) ? 0u : ((sq + 7u) & 7u); }

// Warp w owns units [512 w, 512 w + 512) of the tile and takes them 32 at a time, one per
// lane: staged symbols are read without bank conflicts, patches, counts and block starts
// are read coalesced, and the points of a round are written to consecutive addresses.
// Phase 1 counts each warp's zero symbols in shared memory (the tile's first patch index
// then comes from a chained scan that every tile publishes right after staging); phase 2
// reads the patches and counts once, keeps each unit's repos value (or SFC delta) and count
// in shared memory, and folds the warp's counts, quad / block / repos segments (or SFC
// sums); the block combines the warps, one round of chained scans combines the tiles, and
// the final pass rebuilds every running value with warp scans from its warp's starting
// carry.  A tile holding a value of 2^32 or more or a count of 2^16 or more re-reads them
// in the final pass instead (block mode: never for a stream the encoder wrote, whose repos
// values are 18-bit codes; direct mode: the tile of a cloud's first SFC code, for example).
// With every value below 2^26 as well, the rounds' prefix sums run in 32 bits.
template <bool DIRECT>
__global__ void __launch_bounds__(kThreads, 6) recover_units_kernel(RecoverArgs a) {
    constexpr int kWarps = kThreads / 32;
    __shared__ u8 srep[kTile];
    // block mode: quad symbol q's low 3 bits | 8 (q == 0) | 16 (q == 1) | 32 (block start);
    // the quad index is only used modulo 8, so its running sums need nothing more
    __shared__ u8 squad[DIRECT ? 1 : kTile];
    __shared__ u32 sval[kTile];
    __shared__ u16 scnt[kTile];
    __shared__ u32 slot, wide;
    __shared__ u64 wz[kWarps + 1], wc[kWarps + 1], wd[kWarps + 1];
    __shared__ Seg wq[kWarps + 1], wb[kWarps + 1], wr[kWarps + 1];
    __shared__ u64 base_zero, base_count, base_sfc;
    __shared__ Seg base_quad, base_blk, base_rep;
    __shared__ u8 htab[256];

    const u32 tile = claim_tile(a.tile_counter, &slot);
    const u32 ntiles = gridDim.x;
    const u64 base = (u64)tile * kTile;
    const u32 cnt = (u32)min((u64)kTile, a.units - base);
    const int tid = threadIdx.x;
    const int w = tid >> 5;
    const u32 lane = lane_id();
    const u32 lt = lanemask_lt();
    const bool has_val = a.rep_val != nullptr;
    for (int i = tid; i < 256; i += kThreads) htab[i] = a.hinv ? a.hinv[i] : 0;
    if (tid == 0) wide = 0;
    for (int i = 0; i < kItems; ++i) {
        const u32 e = (u32)i * kThreads + tid;
        if (e < cnt) {
            srep[e] = has_val ? (u8)1 : a.rep_sym[base + e];
            if (!DIRECT) {
                const u32 qs = a.quad_sym[base + e];
                squad[e] = (u8)((qs & 7u) | (qs == 0 ? 8u : 0u) | (qs == 1 ? 16u : 0u) |
                                (a.is_start[base + e] ? 32u : 0u));
            }
        }
    }
    __syncthreads();
    const bool rle = a.rp.rle != 0;
    const u32 wfirst = (u32)w * (32u * kItems);
    SegOp op;

    // repos value of unit e; zc: index of the warp's next patch (advanced on symbol 0).
    // Called by all lanes (it votes).
    auto rep_value = [&](u32 e, bool valid, u64& zc) -> u64 {
        const u32 sym = valid ? srep[e] : 1u;
        const u32 zb = __ballot_sync(kFullMask, valid && !has_val && sym == 0u);
        const u64 z = zc + __popc(zb & lt);
        zc += __popc(zb);
        if (!valid) return 0;
        if (has_val) return a.rep_val[base + e];
        if (sym) return sym - 1u;
        if (z < a.npatch)
            return a.patch32 ? (u64)static_cast<const u32*>(a.rep_patch)[z] : static_cast<const u64*>(a.rep_patch)[z];
        atomicOr(a.err, kErrBadStream);
        return 0;
    };

    // ---- phase 1: zero symbols per warp, chained into the tile's first patch index ----
    if (!has_val) {
        u64 z = 0;
        for (int r = 0; r < kItems; ++r) {
            const u32 e = wfirst + (u32)r * 32u + lane;
            z += __popc(__ballot_sync(kFullMask, e < cnt && srep[e] == 0));
        }
        if (lane == 0) wz[w] = z;
        __syncthreads();
        if (tid == 0) warps_exclusive<kThreads / 32>(wz, 0ull, AddOp{});
        __syncthreads();
        if (w == 0) {
            const u64 r = chain_add(a.status, tile, wz[kWarps], a.err);
            if (tid == 0) base_zero = r;
        }
    } else if (tid < kWarps) {
        wz[tid] = 0;
        if (tid == 0) base_zero = 0;
    }
    __syncthreads();

    // ---- phase 2: values and counts kept; counts, quad, block, repos segments per warp ----
    {
        u64 zc = base_zero + wz[w];
        u64 c = 0, d = 0, bc = 0, rc = 0;
        u32 qc = 0;
        bool any_head = false, any_rhead = false, big = false, w26 = false;
        for (int r = 0; r < kItems; ++r) {
            const u32 e = wfirst + (u32)r * 32u + lane;
            const bool valid = e < cnt;
            const u64 v = rep_value(e, valid, zc);
            const u64 k = rle && valid ? (u64)max(a.counts[base + e], 0) : 0ull;
            c += k;
            if (valid) {
                sval[e] = (u32)v;
                scnt[e] = (u16)k;
                big |= (v >> 32) != 0 || (k >> 16) != 0;
                w26 |= (v >> 26) != 0;
            }
            if (DIRECT) {
                d += v;
            } else {
                const u32 sq = valid ? squad[e] : 16u;
                const bool st = (sq & 32u) != 0;
                const u32 hm = __ballot_sync(kFullMask, st);
                qc = __shfl_sync(kFullMask, warp_seg_incl<u32>(hm, quad_step(sq), qc), 31);
                const u32 bv = st ? a.start_block[base + e] : 0u;
                const u32 last = __shfl_sync(kFullMask, bv, hm ? 31 - __clz(hm) : 0);
                if (hm) bc = last;
                any_head |= hm != 0;
                const u32 hr = __ballot_sync(kFullMask, valid && (st || (sq & 16u) == 0));
                rc = __shfl_sync(kFullMask, warp_seg_incl<u64>(hr, v, rc), 31);
                any_rhead |= hr != 0;
            }
        }
        c = warp_sum(c);
        if (DIRECT) d = warp_sum(d);
        const bool anybig = __any_sync(kFullMask, big), any26 = __any_sync(kFullMask, w26);
        if (lane == 0 && (anybig || any26)) atomicOr(&wide, (anybig ? 1u : 0u) | (any26 ? 2u : 0u));
        if (lane == 0) {
            wc[w] = c;
            wd[w] = d;
            wq[w] = Seg{any_head ? 1ull : 0ull, (u64)qc};
            wb[w] = Seg{any_head ? 1ull : 0ull, bc};
            wr[w] = Seg{any_rhead ? 1ull : 0ull, rc};
        }
    }
    __syncthreads();
    if (tid == 0) {
        warps_exclusive<kThreads / 32>(wc, 0ull, AddOp{});
        if (DIRECT) {
            warps_exclusive<kThreads / 32>(wd, 0ull, AddOp{});
        } else {
            warps_exclusive<kThreads / 32>(wq, Seg{0, 0}, op);
            warps_exclusive<kThreads / 32>(wb, Seg{0, 0}, op);
            warps_exclusive<kThreads / 32>(wr, Seg{0, 0}, op);
        }
    }
    __syncthreads();
    // one warp per chained scan
    if (w == 0) {
        Status* st = a.status + 2 * ntiles;
        if (DIRECT) {
            const u64 r = chain_add(st, tile, wd[kWarps], a.err);
            if (tid == 0) base_sfc = r;
        } else {
            const Seg q = wq[kWarps], b = wb[kWarps], r = wr[kWarps];
            const Pair mine{r.sum, (b.sum & 0xffffffffull) | ((q.sum & 7u) << 32) | (q.head << 35) | (r.head << 36)};
            const Pair p = chain_lookback(st, tile, mine, SegPair{}, a.err);
            if (tid == 0) {
                base_rep = Seg{0, p.lo};
                base_quad = Seg{0, (p.hi >> 32) & 7u};
                base_blk = Seg{0, p.hi & 0xffffffffull};
            }
        }
    } else if (w == 1 && rle) {
        const u64 r = chain_add(a.status + ntiles, tile, wc[kWarps], a.err);
        if (tid == 32) base_count = r;
    }
    if (!rle && tid == 0) base_count = 0;
    __syncthreads();

    // ---- final: coordinates, recover, unshift, expand ----
    const QuantParams q = a.rp.q;
    // block-uniform: values and counts kept in shared memory; and, with every value below 2^26
    // and every count below 2^16, the round's prefix sums fit 32 bits
    const bool kept = (wide & 1u) == 0;
    const bool narrow = wide == 0;
    u64 zc = base_zero + wz[w];
    u64 oc = base_count + wc[w];  // -rle: output position of the warp's first point
    u64 scar = DIRECT ? base_sfc + wd[w] : 0ull;
    u32 qcar = DIRECT ? 0u : (u32)op(base_quad, wq[w]).sum;
    u64 rcar = DIRECT ? 0ull : op(base_rep, wr[w]).sum;
    // corner of the block of the warp's current unit ((blk % nx) * 128, (blk / nx % ny) * 128,
    // (blk / nx / ny) * 128 in u64 arithmetic, kept modulo 2^32 like the cell coordinates they
    // are added to): computed where a block starts, carried to the units after it
    u32 pcx = 0, pcy = 0, pcz = 0;
    auto corner = [&](u64 b, u32& x, u32& y, u32& z) {
        const u64 blk = b < a.nblocks ? a.blk_ids[b] : 0ull;
        const u64 q1 = udiv(blk, a.rp.div_nx), q2 = udiv(q1, a.rp.div_ny);
        x = (u32)((blk - q1 * a.rp.nx) * 128);
        y = (u32)((q1 - q2 * a.rp.ny) * 128);
        z = (u32)(q2 * 128);
    };
    if (!DIRECT) corner(op(base_blk, wb[w]).sum, pcx, pcy, pcz);
    for (int r = 0; r < kItems; ++r) {
        const u32 e = wfirst + (u32)r * 32u + lane;
        const bool valid = e < cnt;
        const u64 rv = kept ? (valid ? (u64)sval[e] : 0ull) : rep_value(e, valid, zc);
        i32 cx = 0, cy = 0, cz = 0;
        if (DIRECT) {
            const u64 sfc = scar + (narrow ? (u64)warp_incl_add((u32)rv) : warp_incl_add(rv));
            scar = __shfl_sync(kFullMask, sfc, 31);
            u32 gx, gy, gz;
            if (a.rp.hilbert) {
                hilbert_xyz(htab, sfc, a.rp.bits, 0u, gx, gy, gz);
            } else {
                gx = gather3(sfc);
                gy = gather3(sfc >> 1);
                gz = gather3(sfc >> 2);
            }
            cx = (i32)gx;
            cy = (i32)gy;
            cz = (i32)gz;
        } else {
            const u32 sq = valid ? squad[e] : 16u;
            const bool st = (sq & 32u) != 0;
            const u32 hm = __ballot_sync(kFullMask, st);
            const u32 quadj = warp_seg_incl<u32>(hm, quad_step(sq), qcar);
            qcar = __shfl_sync(kFullMask, quadj, 31);
            u32 sx = 0, sy = 0, sz = 0;
            if (st) corner(a.start_block[base + e], sx, sy, sz);
            const u32 le = hm & (lt | (1u << lane));
            const int src = le ? 31 - __clz(le) : 0;
            sx = __shfl_sync(kFullMask, sx, src);
            sy = __shfl_sync(kFullMask, sy, src);
            sz = __shfl_sync(kFullMask, sz, src);
            const u32 pbx = le ? sx : pcx, pby = le ? sy : pcy, pbz = le ? sz : pcz;
            pcx = __shfl_sync(kFullMask, pbx, 31);
            pcy = __shfl_sync(kFullMask, pby, 31);
            pcz = __shfl_sync(kFullMask, pbz, 31);
            const u32 hr = __ballot_sync(kFullMask, valid && (st || (sq & 16u) == 0));
            u64 reposj;
            if (narrow) {
                const u32 v32 = (u32)rv, inc = warp_incl_add(v32);
                const u32 lr = hr & (lt | (1u << lane));
                const u32 before = __shfl_sync(kFullMask, inc - v32, lr ? 31 - __clz(lr) : 0);
                reposj = lr ? (u64)(inc - before) : rcar + (u64)inc;
            } else {
                reposj = warp_seg_incl<u64>(hr, rv, rcar);
            }
            rcar = __shfl_sync(kFullMask, reposj, 31);
            if (valid) {
                if (sq & 8u) atomicOr(a.err, kErrBadStream);  // quad patches never occur
                u32 gx, gy, gz;
                if (!a.rp.hilbert) {
                    gx = gather3(reposj);
                    gy = gather3(reposj >> 1);
                    gz = gather3(reposj >> 2);
                } else if (reposj < (1ull << 18)) {
                    hilbert_xyz6(htab, (u32)reposj, a.rp.hstart_inv, gx, gy, gz);
                } else {
                    hilbert_xyz(htab, reposj, 20, 0u, gx, gy, gz);
                }
                cx = (i32)(pbx + ((quadj & 1u) >> 0) * 64u + gx);
                cy = (i32)(pby + ((quadj & 2u) >> 1) * 64u + gy);
                cz = (i32)(pbz + ((quadj & 4u) >> 2) * 64u + gz);
            }
        }
        // -rle: output position from the count prefix; -normal and cells: one per unit.
        u64 c = 1, opos = base + e;
        if (rle) {
            c = !valid ? 0ull : kept ? (u64)scnt[e] : (u64)max(a.counts[base + e], 0);
            const u64 incl = narrow ? (u64)warp_incl_add((u32)c) : warp_incl_add(c);
            opos = oc + incl - c;
            oc += __shfl_sync(kFullMask, incl, 31);
        }
        if (!valid) continue;  // after the round's warp-wide votes and shuffles
        if (a.rp.cells) {
            i32* co = reinterpret_cast<i32*>(a.out);
            co[3 * opos] = cx;
            co[3 * opos + 1] = cy;
            co[3 * opos + 2] = cz;
            continue;
        }
        float x, y, z;
        recover(q, cx, cy, cz, a.rp.off[0], a.rp.off[1], a.rp.off[2], x, y, z);
        if (opos + c > a.nout) {
            atomicOr(a.err, kErrOverflow);
            continue;
        }
        for (u64 k = 0; k < c; ++k) {
            a.out[3 * (opos + k)] = x;
            a.out[3 * (opos + k) + 1] = y;
            a.out[3 * (opos + k) + 2] = z;
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
                          uint64_t base_cnt, int width_cnt, uint64_t nblocks, uint64_t units,
                          unsigned long long* blk_ids, uint8_t* is_start, uint32_t* start_block, ScanStatus status,
                          uint32_t* tile_counter, unsigned long long* count_total, uint32_t* err, cudaStream_t st) {
    const unsigned tiles = (unsigned)((nblocks + kTile - 1) / kTile);
    if (!tiles) return;
    block_streams_kernel<<<tiles, kThreads, 0, st>>>(words_blk, base_blk, width_blk, words_cnt, base_cnt, width_cnt,
                                                     nblocks, units, blk_ids, is_start, start_block, status, tile_counter,
                                                     count_total, err);
}

void launch_fill_u32(uint32_t* p, uint64_t n, uint32_t v, cudaStream_t st) {
    if (n) fill_u32_kernel<<<grid_cap(n), kThreads, 0, st>>>(p, n, v);
}
void launch_fill_u8(uint8_t* p, uint64_t n, uint8_t v, cudaStream_t st) {
    if (n) fill_u8_kernel<<<grid_cap(n), kThreads, 0, st>>>(p, n, v);
}
void launch_count_total(const int32_t* counts, uint64_t n, unsigned long long* total, cudaStream_t st) {
    if (n) count_total_kernel<<<grid_cap(n), kThreads, 0, st>>>(counts, n, total);
}
void launch_recover_units(const RecoverInputs& in, uint64_t units, uint64_t nout, RecoverParams rp,
                          const uint8_t* hilbert_inv_tab, ScanStatus status, uint32_t* tile_counter, float* out, uint32_t* err,
                          cudaStream_t st) {
    RecoverArgs a;
    a.rep_sym = in.rep_sym;
    a.rep_patch = in.rep_patch;
    a.patch32 = in.patch32;
    a.npatch = in.npatch;
    a.quad_sym = in.quad_sym;
    a.is_start = in.is_start;
    a.start_block = in.start_block;
    a.blk_ids = in.blk_ids;
    a.nblocks = in.nblocks;
    a.counts = in.counts;
    a.rep_val = in.rep_val;
    a.units = units;
    a.nout = nout;
    a.rp = rp;
    a.hinv = hilbert_inv_tab;
    a.status = static_cast<Status*>(status);
    a.tile_counter = tile_counter;
    a.out = out;
    a.err = err;
    const unsigned tiles = (unsigned)((units + kTile - 1) / kTile);
    if (!tiles) return;
    if (rp.direct)
        recover_units_kernel<true><<<tiles, kThreads, 0, st>>>(a);
    else
        recover_units_kernel<false><<<tiles, kThreads, 0, st>>>(a);
}

}  // namespace dev
}  // namespace xnyz
