// Stable LSD radix sort of 64-bit keys (optional 32-bit payload), one 8-bit digit per pass,
// single-pass ("onesweep") scatter with decoupled look-back over tiles of 2048, 4096 or 8192 keys;
// up to 8192 keys in one block, all passes in shared memory.
//
// Replaces radix_sort + the per-id std::sort of quantizer/block_quantizer.hpp:33-76 and the
// std::sort of (sfc, index) pairs of composer/block_compressor.hpp:103: the keys packed by
// the key kernels order exactly as (id, reid) resp. (sfc, index) do, and only the digits
// that can be non-zero are sorted.
//
// Per pass: each warp ranks its keys against warp-private digit counters, finding the lanes
// that share a digit with eight ballots, the block turns warp counts into tile-local digit
// offsets, one thread per digit publishes the tile's count (epoch-tagged 64-bit status words, so
// the status array is never cleared between passes), the keys are staged in shared memory in
// digit order, the look-back adds the previous tiles' counts, and the keys are written out in
// coalesced runs.
//
// What bounds it: shared-memory wavefronts (32 per 32 keys: the 8-byte scatter into digit order
// and the counter reads conflict; the peer masks in shared memory of an earlier version took 10
// more) and the look-back, whose length in tiles is the number of tiles in flight.  Measured on
// one B200, 64M random keys, one pass: tiles of 4096 keys (256 threads, 4 blocks per SM) with
// masks 410 us, with ballots 387; tiles of 8192 (512 threads, 2 blocks per SM) 329, 3.1 TB/s of
// 16 B per key.  Persistent blocks that load their next tile's keys early were slower (395): the
// claimed tiles' counts come later, and their successors wait.  Windows of 8 or 16 predecessors
// flood the L2 with status reads (409, 689).
#include "device_common.cuh"
#include "kernels.h"

namespace xnyz {
namespace dev {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kRadix = 256;

// status word: [63:50] epoch, [49:48] flag (1 aggregate, 2 inclusive), [47:0] count
__device__ __forceinline__ u64 pack_status(u32 epoch, u32 flag, u64 count) {
    return ((u64)epoch << 50) | ((u64)flag << 48) | (count & ((1ull << 48) - 1));
}

// Look-back of digit d over the previous tiles' status words, kLookWindow predecessors per
// step (their loads in flight together).  Publishes the tile's inclusive count and returns the
// count of digit d in all previous tiles.
constexpr int kLookWindow = 3;

__device__ __forceinline__ u32 digit_lookback(u64* status, u32 tile, u32 d, u32 count, u32 epoch, u32* err) {
    u32 acc = 0;
    i32 t = (i32)tile - 1;
    u32 spins = 0;
    while (t >= 0) {
        u64 s[kLookWindow];
#pragma unroll
        for (int q = 0; q < kLookWindow; ++q)
            s[q] = t - q >= 0 ? ld_volatile(&status[(u64)(t - q) * kRadix + d]) : 0ull;
        int used = 0;
        bool done = false;
#pragma unroll
        for (int q = 0; q < kLookWindow; ++q) {
            const u32 e = (u32)(s[q] >> 50), f = (u32)(s[q] >> 48) & 3u;
            if (!done && used == q && e == epoch && f != 0) {  // (a word not yet published stops here)
                acc += (u32)s[q];
                ++used;
                done = f == 2;
            }
        }
        if (done) break;
        if (used == 0) {
            if (++spins > kSpinLimit) {
                atomicOr(err, kErrTimeout);
                break;
            }
            if (spins > 8) __nanosleep(32);
        }
        t -= used;
    }
    st_volatile(&status[(u64)tile * kRadix + d], pack_status(epoch, 2, (u64)acc + count));
    return acc;
}

// *p if ok, else 0; volatile, so that all of a thread's loads are issued before its first use of one
// (left to itself the compiler sinks them to their uses for want of registers).
__device__ __forceinline__ u64 load_now(const u64* p, bool ok) {
    u64 v;
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.b64 %0, 0; @q ld.global.b64 %0, [%1]; }"
                 : "=&l"(v)
                 : "l"(p), "r"((u32)ok));
    return v;
}

// Byte `shift / 8` of a key.  volatile: extracted again where needed instead of kept in a register.
struct DigitOf {
    u32 sel;
    __device__ __forceinline__ explicit DigitOf(int shift) : sel(0x4440u | ((u32)shift >> 3)) {}
    __device__ __forceinline__ u32 operator()(u64 key) const {
        u32 d;
        asm volatile("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"((u32)key), "r"((u32)(key >> 32)), "r"(sel));
        return d & 255u;
    }
};

// Ranks of a warp's keys (ITEMS per lane, key i of lane l is the warp's 32 i + l-th) among its keys
// of the same digit, two 16-bit ranks per register; wh (zeroed) receives the warp's digit counts.
template <int ITEMS>
__device__ __forceinline__ void warp_ranks(const u64 (&k)[ITEMS], u32 first, u32 cnt, const DigitOf& digit, u32* wh,
                                           u32 (&rank2)[(ITEMS + 1) / 2]) {
    const u32 lt = lanemask_lt();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const bool ok = first + 32u * i < cnt;
        const u32 d = digit(k[i]);
        u32 peers = __ballot_sync(kFullMask, ok);  // the lanes with my digit: one ballot per bit
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            u32 m;
            asm("{ .reg .pred p; and.b32 %0, %1, %2; setp.ne.u32 p, %0, 0; vote.sync.ballot.b32 %0, p, 0xffffffff; "
                "@!p not.b32 %0, %0; }"
                : "=&r"(m)
                : "r"(d), "r"(1u << b));
            peers &= m;
        }
        const u32 below = peers & lt;
        const u32 prev = ok ? wh[d] : 0u;
        __syncwarp();
        if (ok && below == 0u) wh[d] = prev + __popc(peers);
        __syncwarp();
        const u32 rank = prev + __popc(below);
        if (i & 1) rank2[i / 2] |= rank << 16;
        else rank2[i / 2] = rank;
    }
}

// What the digit columns' scan keeps in shared memory besides the warps' counters.
struct ScanShared {
    u32 wsum[kRadix / 32], lower[kRadix], upper[kRadix], count[kRadix], start[kRadix];
};

// Turns the warps' digit counts into the tile positions of each warp's first key of each digit.
// Threads d and d + 256 take digit d, each over half of the warps.  publish(digit, count) is called
// by thread `digit` as soon as the tile's count is known.  sh.count keeps the digits' counts, sh.start (+ the
// earlier wsum) their first tile positions.  Ends with a barrier.
template <typename F>
__device__ __forceinline__ void digit_starts(u32* whist, ScanShared& sh, F&& publish) {
    const int tid = threadIdx.x;
    const u32 d = (u32)tid & (kRadix - 1), lane = lane_id();
    u32* col = whist + (tid >> 8) * (kWarps / 2) * kRadix + d;
    u32 half = 0;
#pragma unroll
    for (int ww = 0; ww < kWarps / 2; ++ww) half += col[ww * kRadix];
    if (tid >= kRadix) sh.upper[d] = half;
    else sh.lower[d] = half;
    __syncthreads();
    if (tid < kRadix) {
        const u32 c = half + sh.upper[d];
        publish(d, c);
        const u32 incl = warp_incl_add(c);
        if (lane == 31) sh.wsum[tid >> 5] = incl;
        sh.count[d] = c;
        sh.start[d] = incl - c;
    }
    __syncthreads();
    u32 start = sh.start[d];
    for (u32 ww = 0; ww < (d >> 5); ++ww) start += sh.wsum[ww];
    u32 run = start + (tid >= kRadix ? sh.lower[d] : 0u);
#pragma unroll
    for (int ww = 0; ww < kWarps / 2; ++ww) {
        const u32 c = col[ww * kRadix];
        col[ww * kRadix] = run;
        run += c;
    }
    __syncthreads();
}

// One tile per block.  Positions within the array fit 32 bits (n < 2^31).  Keys only: 2 blocks per
// SM (64 registers, 82 KB shared for 16 keys per thread); with payload: 1.
template <bool PAYLOAD, int ITEMS>
__global__ void __launch_bounds__(kThreads, PAYLOAD ? 1 : 2) sort_pass_kernel(const u64* __restrict__ kin, u64* __restrict__ kout,
                                                             const u32* __restrict__ vin, u32* __restrict__ vout,
                                                             u32 n, int shift, const u32* __restrict__ offsets,
                                                             u64* status, u32 epoch, u32* tile_counter, u32* err) {
    constexpr u32 kTile = kThreads * ITEMS;
    extern __shared__ __align__(16) unsigned char smem[];
    u64* skeys = reinterpret_cast<u64*>(smem);           // kTile
    u32* whist = reinterpret_cast<u32*>(skeys + kTile);  // kWarps * kRadix
    u32* svals = whist + kWarps * kRadix;                // kTile (PAYLOAD)
    __shared__ ScanShared sh;
    __shared__ u32 gbase[kRadix];
    __shared__ u32 slot;
    const int tid = threadIdx.x, w = tid >> 5, lane = lane_id();
    if (tid == 0) slot = atomicAdd(tile_counter, 1u);  // claimed in launch order (claim_tile)
    u32* wh = whist + w * kRadix;
#pragma unroll
    for (int i = 0; i < kRadix / 32; ++i) wh[i * 32 + lane] = 0u;
    __syncthreads();
    const u32 tile = slot;
    const u32 first = (u32)w * (32 * ITEMS) + lane;  // my first key in the tile; then every 32nd
    const u32 cnt = min(kTile, n - tile * kTile);
    const DigitOf digit(shift);
    u64 k[ITEMS];
    u32 v[ITEMS];
    {
        const u64* kp = kin + (u64)tile * kTile + first;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) k[i] = load_now(kp + 32 * i, first + 32u * i < cnt);
        if (PAYLOAD) {
            const u32* vp = vin + (u64)tile * kTile + first;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) v[i] = first + 32u * i < cnt ? vp[32 * i] : 0u;
        }
    }
    u32 rank2[(ITEMS + 1) / 2];
    warp_ranks<ITEMS>(k, first, cnt, digit, wh, rank2);
    __syncthreads();
    digit_starts(whist, sh, [&](u32 d, u32 c) {
        st_volatile(&status[(u64)tile * kRadix + d], pack_status(epoch, tile == 0 ? 2 : 1, c));
    });
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (first + 32u * i < cnt) {
            const u32 p = wh[digit(k[i])] + ((rank2[i / 2] >> (16 * (i & 1))) & 0xffffu);
            skeys[p] = k[i];
            if (PAYLOAD) svals[p] = v[i];
        }
    }
    if (tid < kRadix) {
        const u32 before = tile == 0 ? 0u : digit_lookback(status, tile, (u32)tid, sh.count[tid], epoch, err);
        u32 start = sh.start[tid];
        for (u32 ww = 0; ww < ((u32)tid >> 5); ++ww) start += sh.wsum[ww];
        gbase[tid] = offsets[tid] + before - start;  // + tile slot p: the output position (wrapping)
    }
    __syncthreads();

#pragma unroll 4
    for (u32 p = (u32)tid; p < cnt; p += kThreads) {
        const u64 key = skeys[p];
        const u32 o = gbase[digit(key)] + p;
        if (o < n) {
            kout[o] = key;
            if (PAYLOAD) vout[o] = svals[p];
        } else {  // only after an expired look-back wait: flagged, never written
            atomicOr(err, kErrPlacement);
        }
    }
}

// Up to kThreads * ITEMS keys: one block, the keys in shared memory from the first pass to the last
// (no launches, look-back or trips through global memory between passes: 5 passes over 1013 keys
// 53 -> 17 us, over 8000 keys 58 -> 34).
template <bool PAYLOAD, int ITEMS>
__global__ void __launch_bounds__(kThreads) sort_small_kernel(const u64* kin, u64* kout, const u32* vin, u32* vout, u32 n,
                                                              int passes) {
    constexpr u32 kTile = kThreads * ITEMS;
    extern __shared__ __align__(16) unsigned char smem[];
    u64* skeys = reinterpret_cast<u64*>(smem);           // kTile
    u32* whist = reinterpret_cast<u32*>(skeys + kTile);  // kWarps * kRadix
    u32* svals = whist + kWarps * kRadix;                // kTile (PAYLOAD)
    __shared__ ScanShared sh;
    const int tid = threadIdx.x, w = tid >> 5, lane = lane_id();
    u32* wh = whist + w * kRadix;
    const u32 first = (u32)w * (32 * ITEMS) + lane;
    u64 k[ITEMS];
    u32 v[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const u32 e = first + 32u * i;
        k[i] = e < n ? kin[e] : 0ull;
        if (PAYLOAD) v[i] = e < n ? vin[e] : 0u;
    }
    for (int p = 0; p < passes; ++p) {
        const DigitOf digit(8 * p);
#pragma unroll
        for (int i = 0; i < kRadix / 32; ++i) wh[i * 32 + lane] = 0u;
        __syncwarp();
        u32 rank2[(ITEMS + 1) / 2];
        warp_ranks<ITEMS>(k, first, n, digit, wh, rank2);
        __syncthreads();
        digit_starts(whist, sh, [](u32, u32) {});
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (first + 32u * i < n) {
                const u32 at = wh[digit(k[i])] + ((rank2[i / 2] >> (16 * (i & 1))) & 0xffffu);
                skeys[at] = k[i];
                if (PAYLOAD) svals[at] = v[i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const u32 e = first + 32u * i;
            if (e < n) {
                k[i] = skeys[e];
                if (PAYLOAD) v[i] = svals[e];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const u32 e = first + 32u * i;
        if (e < n) {
            kout[e] = k[i];
            if (PAYLOAD) vout[e] = v[i];
        }
    }
}

constexpr int smem_bytes(bool payload, int items) {
    return kThreads * items * (payload ? 12 : 8) + kWarps * kRadix * 4;
}

template <bool PAYLOAD, int ITEMS>
void launch_pass(const u64* kin, u64* kout, const u32* vin, u32* vout, u32 n, int shift, const u32* offsets, u64* status,
                 u32 epoch, u32* tile_counter, u32* err, cudaStream_t st) {
    // The dynamic shared-memory limit is a per-device function attribute; setting it on
    // every launch keeps multi-device use correct and costs a few microseconds.
    constexpr int smem = smem_bytes(PAYLOAD, ITEMS);
    if (smem > 40 << 10)
        cudaFuncSetAttribute(sort_pass_kernel<PAYLOAD, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const u32 tiles = (n + kThreads * ITEMS - 1) / (kThreads * ITEMS);
    sort_pass_kernel<PAYLOAD, ITEMS><<<tiles, kThreads, smem, st>>>(kin, kout, vin, vout, n, shift, offsets, status,
                                                                    epoch, tile_counter, err);
}

template <bool PAYLOAD, int ITEMS>
void launch_small(const u64* kin, u64* kout, const u32* vin, u32* vout, u32 n, int passes, cudaStream_t st) {
    constexpr int smem = smem_bytes(PAYLOAD, ITEMS);
    if (smem > 40 << 10)
        cudaFuncSetAttribute(sort_small_kernel<PAYLOAD, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    sort_small_kernel<PAYLOAD, ITEMS><<<1, kThreads, smem, st>>>(kin, kout, vin, vout, n, passes);
}

__global__ void __launch_bounds__(256) histogram_kernel(const u64* __restrict__ keys, u64 n, int passes,
                                                             u32* hist) {
    __shared__ u32 sh[8 * kRadix];
    for (int i = threadIdx.x; i < passes * kRadix; i += 256) sh[i] = 0;
    __syncthreads();
    const u64 stride = (u64)gridDim.x * 256;
    for (u64 j = (u64)blockIdx.x * 256 + threadIdx.x; j < n; j += stride) {
        const u64 key = keys[j];
        for (int p = 0; p < passes; ++p) atomicAdd(&sh[p * kRadix + (u32)((key >> (8 * p)) & 255u)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kRadix; i += 256)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// One block per pass: digit counts -> exclusive digit offsets, in place.
__global__ void __launch_bounds__(kRadix) offsets_kernel(u32* hist) {
    __shared__ u32 scratch[16];
    u32* h = hist + blockIdx.x * kRadix;
    const u32 c = h[threadIdx.x];
    u32 total;
    const u32 e = block_exclusive<kRadix>(c, 0u, AddOp{}, scratch, total);
    h[threadIdx.x] = e;
}

}  // namespace

void launch_sort_histogram(const unsigned long long* keys, uint64_t n, int passes, uint32_t* hist, cudaStream_t st) {
    u64 blocks = (n + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    if (blocks < 1) blocks = 1;
    histogram_kernel<<<(unsigned)blocks, 256, 0, st>>>(keys, n, passes, hist);
}

void launch_sort_offsets(uint32_t* hist, int passes, cudaStream_t st) {
    offsets_kernel<<<passes, kRadix, 0, st>>>(hist);
}

void launch_sort_pass(const unsigned long long* kin, unsigned long long* kout, const uint32_t* vin, uint32_t* vout,
                      uint64_t n, int shift, const uint32_t* offsets, unsigned long long* status, uint32_t epoch,
                      uint32_t* tile_counter, uint32_t* err, cudaStream_t st) {
    if (!n) return;
    const u32 m = (u32)n;
#define XNYZ_PASS(P, I) launch_pass<P, I>(kin, kout, vin, vout, m, shift, offsets, status, epoch, tile_counter, err, st)
    switch (sort_tile(n) / kThreads) {
        case 4: vin ? XNYZ_PASS(true, 4) : XNYZ_PASS(false, 4); break;
        case 8: vin ? XNYZ_PASS(true, 8) : XNYZ_PASS(false, 8); break;
        default: vin ? XNYZ_PASS(true, 16) : XNYZ_PASS(false, 16); break;
    }
#undef XNYZ_PASS
}

void launch_sort_small(const unsigned long long* kin, unsigned long long* kout, const uint32_t* vin, uint32_t* vout,
                       uint64_t n, int passes, cudaStream_t st) {
    const u32 m = (u32)n;
    if (n <= 4 * kThreads)
        vin ? launch_small<true, 4>(kin, kout, vin, vout, m, passes, st) : launch_small<false, 4>(kin, kout, vin, vout, m, passes, st);
    else
        vin ? launch_small<true, 16>(kin, kout, vin, vout, m, passes, st) : launch_small<false, 16>(kin, kout, vin, vout, m, passes, st);
}

}  // namespace dev
}  // namespace xnyz
