// Parallel decoding of one unindexed prefix-code stream: Huffman (huffman_encoder.hpp:205-243),
// Golomb-Rice (golomb_rice_encoder.hpp:150-192) and exp-Golomb (huffman_encoder.hpp:398-442).
// The streams carry no sync points.  decode_sync_kernel decodes from guessed entries and corrects
// them; streams that do not fall in step go to decode_stream_kernel, whose work does not depend
// on that.  Both are exact for any prefix code.  The entry-table decoder:
//
//   1. every thread owns one S-bit subsequence and computes, for each entry offset e < L
//      (L = longest codeword; Golomb-Rice: k + 2 classes), where decoding from there leaves
//      the subsequence and how many codewords start inside.  Chains that reach a codeword
//      start of one of R recorded root chains reuse its result (the roots' codeword starts
//      are kept as bitmaps over the first WIN bits);
//   2. warp 0 composes the block's T transition tables;
//   3. blocks resolve their true entry offset by decoupled look-back over the predecessors'
//      composed tables (function composition with warp shuffles);
//   4. lane 0 walks the block's tables from the true entry (entries a table does not cover,
//      after a codeword longer than L crossed a boundary, are decoded on the spot);
//   5. every thread decodes its subsequence once from its true entry and stores the symbols.
//
// The block's stream words (plus a halo) and the Huffman primary table are staged in shared
// memory; codewords are read through a 64-bit register bit buffer refilled one word at a
// time.  Waits are bounded (kSpinLimit): a block that gives up sets the host's fallback flag and
// returns; that is no error yet, since the host then has one thread decode the stream.
#include "device_common.cuh"
#include "kernels.h"

namespace xnyz {
namespace dev {

namespace {

constexpr int T = kDecodeBlockSubs;     // subsequences (threads) per block
constexpr int HALO = 8;                 // words staged after the block's range
// Subsequence geometry per code: bits per subsequence, staged words per block.
template <int KIND>
struct Geo {
    static constexpr int S = KIND == kCodeGolombRice ? kDecodeSubBitsGR : kDecodeSubBits;
    static constexpr int STAGED = T * S / 32 + HALO;
};
constexpr int WIN = 256;                // root bitmaps cover codeword starts in [0, WIN)
constexpr int WINW = WIN / 32;
constexpr int R = 3;                    // recorded root chains per subsequence
constexpr int kMaxL = kDecodeMaxL;
constexpr int kMaxRootBits = 11;
constexpr u32 kOOD = 0xffu;             // exit outside the next subsequence's entry range
constexpr u64 kFar = 1ull << 20;        // length given to an invalid Huffman code: ends the chain
// Why the host has to decode a stream otherwise (kernels.h: launch_decode_sync).
constexpr u32 kWaitExpired = 1u;
constexpr u32 kNotConverged = 2u;
constexpr u32 kWideValue = 4u;
static_assert(kDecodeSubBits % 32 == 0 && kDecodeSubBitsGR % 32 == 0 && T % 32 == 0 && T <= 1024 &&
                  WIN <= kDecodeSubBits && WIN <= kDecodeSubBitsGR && kDecodeSubBits <= kDecodeSubBitsGR,
              "decode geometry");

// ------------------------------------------------------------- stream source ----------
// A stream starts `base` (< 32) bits into `g`.  Word k of `g` is read from shared memory
// when staged, else from global memory; words past the stream read as zero.
struct Src {
    const u32* g;
    u32 base;
    u64 total_bits;
    u64 nwords;
    const u32* sm;
    u64 sm_w0;
    u64 staged;  // words in sm
    __device__ __forceinline__ u32 word(u64 k) const {
        const u64 d = k - sm_w0;
        if (d < staged) return sm[d];
        return k < nwords ? __ldg(g + k) : 0u;
    }
    __device__ __forceinline__ u32 word_be(u64 k) const { return __byte_perm(word(k), 0, 0x0123); }
    // 32 bits of the MSB-first stream from stream bit p, first bit in bit 31.
    __device__ __forceinline__ u32 msb32(u64 p) const {
        const u64 q = base + p;
        const u32 o = (u32)(q & 31u);
        const u32 a = word_be(q >> 5);
        return o ? ((a << o) | (word_be((q >> 5) + 1) >> (32u - o))) : a;
    }
    // 64 bits of the LSB-first stream from stream bit p, first bit in bit 0.
    __device__ __forceinline__ u64 lsb64(u64 p) const {
        const u64 q = base + p;
        const u32 o = (u32)(q & 31u);
        const u64 k = q >> 5;
        const u64 lo = (u64)word(k) | ((u64)word(k + 1) << 32);
        return o ? ((lo >> o) | ((u64)word(k + 2) << (64u - o))) : lo;
    }
};

// MSB-first bit buffer: the next bit is bit 63 of buf, nb bits are valid, the rest are 0.
struct MsbReader {
    u64 buf;
    int nb;
    u64 wk;
    __device__ __forceinline__ void init(const Src& s, u64 p) {
        const u64 q = s.base + p;
        wk = q >> 5;
        const u32 o = (u32)(q & 31u);
        buf = (((u64)s.word_be(wk) << 32) | (u64)s.word_be(wk + 1)) << o;
        nb = 64 - (int)o;
        wk += 2;
    }
    __device__ __forceinline__ void refill(const Src& s) {
        if (nb <= 32) {
            buf |= (u64)s.word_be(wk) << (32 - nb);
            nb += 32;
            ++wk;
        }
    }
    __device__ __forceinline__ void skip(int n) {
        buf = n >= 64 ? 0ull : buf << n;
        nb -= n;
    }
};

// LSB-first bit buffer: the next bit is bit 0 of buf.
struct LsbReader {
    u64 buf;
    int nb;
    u64 wk;
    __device__ __forceinline__ void init(const Src& s, u64 p) {
        const u64 q = s.base + p;
        wk = q >> 5;
        const u32 o = (u32)(q & 31u);
        buf = ((u64)s.word(wk) | ((u64)s.word(wk + 1) << 32)) >> o;
        nb = 64 - (int)o;
        wk += 2;
    }
    __device__ __forceinline__ void refill(const Src& s) {
        if (nb <= 32) {
            buf |= (u64)s.word(wk) << nb;
            nb += 32;
            ++wk;
        }
    }
    __device__ __forceinline__ void skip(int n) {
        buf = n >= 64 ? 0ull : buf >> n;
        nb -= n;
    }
};

// ------------------------------------------------------------- codewords --------------
struct Code {
    const u32* root;   // primary table (shared memory when staged)
    const u32* tree;   // global
    const u64* symvals;  // null: table entries hold the symbol values themselves
    int rb;
    int k;
    int zigzag;
};

// Huffman from a 32-bit window: primary lookup, tree walk for codes longer than rb.
// Returns the length (0: no code) and the entry payload (symbol value or index).
__device__ __forceinline__ u32 huff_lookup(const Code& c, u32 top, u32& sym) {
    const u32 e = c.root[top >> (32 - c.rb)];
    if (!(e & 0x80000000u)) {
        sym = e & 0xffffffu;
        return e >> 24;
    }
    u32 node = e & 0x7fffffffu;
    for (u32 i = (u32)c.rb; i < 32u; ++i) {
        const u32 ch = __ldg(&c.tree[2 * node + ((top >> (31u - i)) & 1u)]);
        if (ch & 0x80000000u) {
            sym = ch & 0x7fffffffu;
            return ch == 0xffffffffu ? 0u : i + 1;
        }
        node = ch;
    }
    sym = 0;
    return 0;
}

// Golomb-Rice codeword at stream bit p without the bit buffer (long runs, large k).
// A codeword that does not end inside the stream returns total_bits + 1 - p.
__device__ u64 gr_generic(const Src& s, u64 p, int k, u64& val) {
    u64 q = 0;
    u64 v = s.lsb64(p);
    while (v == ~0ull) {
        q += 64;
        if (p + q >= s.total_bits + 64) {
            val = 0;
            return s.total_bits + 1 - p;
        }
        v = s.lsb64(p + q);
    }
    q += (u64)(__ffsll((long long)~v) - 1);
    if (p + q + 1 + (u64)k > s.total_bits) {
        val = 0;
        return s.total_bits + 1 - p;
    }
    const u64 r = k ? (s.lsb64(p + q + 1) & ((1ull << k) - 1)) : 0ull;
    val = (q << k) + r;
    return q + 1 + (u64)k;
}

// exp-Golomb codeword at stream bit p without the bit buffer.
__device__ u64 eg_generic(const Src& s, u64 p, int k, int zigzag, u64& val) {
    u64 z = 0;
    u32 w = s.msb32(p);
    while (w == 0u) {
        z += 32;
        if (p + z >= s.total_bits + 64) {
            val = 0;
            return s.total_bits + 1 - p;
        }
        w = s.msb32(p + z);
    }
    z += (u64)__clz((int)w);
    if (p + 2 * z + 1 + (u64)k > s.total_bits) {
        val = 0;
        return s.total_bits + 1 - p;
    }
    u64 n1;
    if (z + 1 <= 32) {
        n1 = s.msb32(p + z) >> (31 - z);
    } else {
        const u64 hi = s.msb32(p + z), lo = s.msb32(p + z + 32);
        n1 = z + 1 >= 64 ? ~0ull : (((hi << 32) | lo) >> (63 - z));
    }
    const u64 rbits = k ? (s.msb32(p + 2 * z + 1) >> (32 - k)) : 0ull;
    const u64 low = k ? (u64)(__brev((u32)rbits) >> (32 - k)) : 0ull;
    const u64 u = ((n1 - 1) << k) | low;
    val = zigzag ? ((u >> 1) ^ (~(u & 1ull) + 1ull)) : u;
    return 2 * z + 1 + (u64)k;
}

// One codeword through the bit buffer at stream bit p (the reader is positioned at p).
// Returns the length; Huffman returns kFar for a prefix that is no code.  `val` is the
// symbol value (Huffman: the table payload, mapped through symvals when present).
template <int KIND>
struct Dec;

template <>
struct Dec<kCodeHuffman> {
    MsbReader r;
    __device__ __forceinline__ void init(const Src& s, u64 p) { r.init(s, p); }
    __device__ __forceinline__ u64 step(const Src& s, const Code& c, u64, u64& val, bool want) {
        r.refill(s);
        u32 sym;
        const u32 len = huff_lookup(c, (u32)(r.buf >> 32), sym);
        if (!len) {
            val = 0;
            return kFar;
        }
        r.skip((int)len);
        if (want) val = c.symvals ? __ldg(&c.symvals[sym]) : (u64)sym;
        return len;
    }
};

template <>
struct Dec<kCodeGolombRice> {
    LsbReader r;
    __device__ __forceinline__ void init(const Src& s, u64 p) { r.init(s, p); }
    __device__ __forceinline__ u64 step(const Src& s, const Code& c, u64 p, u64& val, bool) {
        r.refill(s);
        const int k = c.k;
        if (r.buf != ~0ull) {
            const int t = __ffsll((long long)~r.buf) - 1;
            if (t < r.nb && t + 1 + k <= r.nb) {
                const u64 rem = k ? ((r.buf >> (t + 1)) & ((1ull << k) - 1)) : 0ull;
                val = ((u64)t << k) | rem;
                const int len = t + 1 + k;
                r.skip(len);
                return (u64)len;
            }
        }
        const u64 len = gr_generic(s, p, k, val);
        r.init(s, p + len);
        return len;
    }
};

template <>
struct Dec<kCodeExpGolomb> {
    MsbReader r;
    __device__ __forceinline__ void init(const Src& s, u64 p) { r.init(s, p); }
    __device__ __forceinline__ u64 step(const Src& s, const Code& c, u64 p, u64& val, bool) {
        r.refill(s);
        const int k = c.k;
        if (r.buf) {
            const int z = __clzll((long long)r.buf);
            const int len = 2 * z + 1 + k;
            if (z < r.nb && len <= r.nb) {
                const u64 n1 = (r.buf << z) >> (63 - z);
                const u64 rbits = k ? ((r.buf << (2 * z + 1)) >> (64 - k)) : 0ull;
                const u64 low = k ? (u64)(__brev((u32)rbits) >> (32 - k)) : 0ull;
                const u64 u = ((n1 - 1) << k) | low;
                val = c.zigzag ? ((u >> 1) ^ (~(u & 1ull) + 1ull)) : u;
                r.skip(len);
                return (u64)len;
            }
        }
        const u64 len = eg_generic(s, p, k, c.zigzag, val);
        r.init(s, p + len);
        return len;
    }
};

// One codeword at p without a persistent reader (the on-the-spot walks of step 4).
template <int KIND>
__device__ __forceinline__ u64 codeword_at(const Src& s, const Code& c, u64 p, u64& val) {
    Dec<KIND> d;
    d.init(s, p);
    return d.step(s, c, p, val, false);
}

// One-bits of an LSB-first stream from stream bit p up to the first zero.
__device__ u64 lead_ones(const Src& s, u64 p) {
    u64 q = 0;
    while (p + q < s.total_bits) {
        const u64 v = s.lsb64(p + q);
        if (v != ~0ull) return q + (u64)(__ffsll((long long)~v) - 1);
        q += 64;
    }
    return q;
}

// Entry classes.  Golomb-Rice: a codeword crossing into subsequence s ends at an offset
// x <= k, or its terminating zero lies inside s after a run of ones that reaches back to
// s's first bit, so x = k + 1 + (leading ones of s): k + 2 classes, the last one "special".
// Other codes: offsets 0 .. L-1.
template <int KIND>
__device__ __forceinline__ u32 entry_index(u64 x, int L, int k) {
    if (KIND == kCodeGolombRice) return x <= (u64)k ? (u32)x : (u32)(k + 1);
    return x < (u64)L ? (u32)x : kOOD;
}
template <int KIND>
__device__ __forceinline__ u64 entry_offset(const Src& s, u32 i, u64 Bsub, int k) {
    if (KIND == kCodeGolombRice && i == (u32)(k + 1)) return (u64)k + 1 + lead_ones(s, Bsub);
    return i;
}

// Golomb-Rice transition table of one subsequence [B, Bend) by lockstep simulation.  The
// codeword-start map f(s) = z(s) + 1 + k (z(s): first zero bit at or after s) is monotone, so
// the chains of entries 0..k keep their order, merge when they land on one position, and at
// step n all lie within codeword n of entry 0's chain.  While that codeword is shorter than
// 64 bits (k <= 30 and a unary part below 64 - k - 1 bits), the active chains are a 64-bit
// position mask over a shared 128-bit zero window, and their entries a boundary mask over
// 0..k.  Entry k + 1 (a unary run crossing B) is entry 0's chain after its first codeword.
// Called by every thread of the warp (valid: this thread owns a subsequence); the loops are
// warp-uniform (__any_sync) so that lanes with different chain counts stay converged.
// Returns false (table incomplete) when a codeword is too long for the masks or the stream
// ends within reach; the caller then runs the generic loop.
__device__ bool gr_lockstep_table(const Src& src, u64 B, u64 Bend, int k, u32* tab, int t, bool valid) {
    constexpr int S = Geo<kCodeGolombRice>::S;
    const u32 span = valid ? (u32)(Bend - B) : 0u;
    const bool full = span == (u32)S;
    // near the end of the stream codewords may run past it (the generic decoder gives those
    // a length that ends the chain): left to the generic loop
    bool ok = valid && B + span + 192 <= src.total_bits;
    const int ne = min(k + 1, (int)span);  // entries with a codeword start inside
    if (ok)
        for (int e = ne; e <= k; ++e) tab[e * T + t] = kOOD;  // (only in a short last subsequence)
    u64 act = ok ? (ne >= 64 ? ~0ull : ((1ull << ne) - 1ull)) : 0ull;  // group positions - base
    u64 gb = act;     // first entry of every group
    u64 alive = act;  // entries not yet recorded
    u32 base = 0, n = 0, exit0 = kOOD, count0 = 0;
    // The 128 bits from B + base, kept in five stream words that move forward with base (the
    // groups only advance), instead of two six-word reads per step.
    u64 wk = (src.base + B) >> 5;
    u32 wv[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) wv[i] = src.word(wk + i);
    while (__any_sync(kFullMask, act != 0ull)) {
        u64 z0 = 0, z1 = 0;
        if (act) {
            const u64 q = src.base + B + base;
            const u64 kk = q >> 5;
            if (kk - wk >= 5) {
                wk = kk;
#pragma unroll
                for (int i = 0; i < 5; ++i) wv[i] = src.word(wk + i);
            } else {
                while (wk < kk) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) wv[i] = wv[i + 1];
                    wv[4] = src.word(wk + 5);
                    ++wk;
                }
            }
            const u32 o = (u32)(q & 31u);
            const u64 a = (u64)wv[0] | ((u64)wv[1] << 32), b = (u64)wv[2] | ((u64)wv[3] << 32);
            z0 = ~(o ? (a >> o) | (b << (64u - o)) : a);
            z1 = ~(o ? (b >> o) | ((u64)wv[4] << (64u - o)) : b);
            ++n;
        }
        // successors, in order; groups landing on the previous group's position merge
        u64 a = act, g = gb, nact = 0, ngb = gb;
        u32 first_s = 0, prev_s = 0xffffffffu;
        bool any = false;
        while (__any_sync(kFullMask, a != 0ull)) {
            if (!a) continue;
            const int j = __ffsll((long long)a) - 1;
            a &= a - 1;
            const int e0 = __ffsll((long long)g) - 1;
            g &= g - 1;
            u32 zp = 0;
            if (z0 >> j) {
                zp = base + (u32)j + (u32)(__ffsll((long long)(z0 >> j)) - 1);
            } else if (z1) {
                zp = base + 64u + (u32)(__ffsll((long long)z1) - 1);
            } else {  // a unary run longer than the window
                ok = false;
                a = 0;
                continue;
            }
            const u32 sp = zp + 1u + (u32)k;
            if (sp == prev_s) {
                ngb &= ~(1ull << e0);
                continue;
            }
            if (!any) {
                first_s = sp;
                any = true;
            }
            if (sp - first_s >= 64u) {  // the chains span more than 64 bits
                ok = false;
                a = 0;
                continue;
            }
            nact |= 1ull << (sp - first_s);
            prev_s = sp;
        }
        if (!ok) {
            act = 0;
            continue;
        }
        if (!act) continue;
        act = nact;
        gb = ngb;
        base = first_s;
        // groups at or past the end leave: they are the top groups, entries from their first
        // entry up to the next group's first entry (or the last alive entry)
        const u32 lo = span > base ? span - base : 0u;  // first leaving bit
        const u64 leave = lo >= 64 ? 0ull : (act >> lo) << lo;
        if (leave) {
            u64 a2 = act, g2 = gb;
            while (a2) {
                const int j = __ffsll((long long)a2) - 1;
                a2 &= a2 - 1;
                const int e0 = __ffsll((long long)g2) - 1;
                g2 &= g2 - 1;
                if (!((leave >> j) & 1ull)) continue;
                const int e1 = g2 ? __ffsll((long long)g2) - 1 : 64;  // next group's first entry
                const u32 P = base + (u32)j;
                const u32 ox = full ? entry_index<kCodeGolombRice>((u64)P - S, k + 2, k) : kOOD;
                const u64 below1 = e1 >= 64 ? ~0ull : ((1ull << e1) - 1ull), below0 = (1ull << e0) - 1ull;
                u64 m = alive & below1 & ~below0;
                while (m) {
                    const int e = __ffsll((long long)m) - 1;
                    m &= m - 1;
                    tab[e * T + t] = ox | (n << 8);
                    if (e == 0) {
                        exit0 = ox;
                        count0 = n;
                    }
                }
                alive &= ~below1 | below0;
            }
            act &= ~leave;
            gb &= alive;
        }
    }
    if (ok) tab[(k + 1) * T + t] = exit0 | ((count0 - 1u) << 8);
    return ok;
}

struct Args {
    const u32* words;
    u32 base;
    u64 total_bits;
    u64 nsub;
    int L;
    Code code;
    const u32* root_global;
    u64 nsym;
    int out_width;
    void* out;
    u32* flag;
    u64* agg;   // [tile][kMaxL]: exit | count << 8
    u64* inc;   // [tile][2]: exit, count through the tile
    u32* tile_counter;
    u32* err;
    u32* need_fallback;
    unsigned long long* total_codewords;
};

// Shared memory: scount[T] u64 | sw[STAGED] | bm[R][WINW][T] | sstart[T] | slot | tab[L][T] | root[2^rb]
template <int KIND>
__host__ __device__ constexpr size_t smem_for(int L, int rb) {
    return 8 * T + 4 * (Geo<KIND>::STAGED + R * WINW * T + T + 4) + 4ull * L * T + (rb ? 4ull << rb : 0);
}

// Output of symbols: u8 streams pack four symbols per 32-bit store where a word lies inside
// the thread's range.
struct ByteOut {
    u8* out;
    u64 first;
    u32 acc;
    __device__ __forceinline__ void put(u64 i, u64 v) {
        const u32 sh = (u32)(i & 3u) * 8u;
        acc = (sh ? acc : 0u) | ((u32)(v & 0xffu) << sh);
        if (sh == 24u) {
            const u64 w0 = i & ~3ull;
            if (w0 >= first) {
                *reinterpret_cast<u32*>(out + w0) = acc;
            } else {
                for (u64 j = first; j <= i; ++j) out[j] = (u8)(acc >> ((j & 3u) * 8u));
            }
        }
    }
    __device__ __forceinline__ void flush(u64 end) {  // symbols [.., end) were put
        if (end & 3u) {
            const u64 w0 = end & ~3ull;
            for (u64 j = w0 > first ? w0 : first; j < end; ++j) out[j] = (u8)(acc >> ((j & 3u) * 8u));
        }
    }
};

template <int KIND>
__global__ void __launch_bounds__(T) decode_stream_kernel(Args a) {
    constexpr int S = Geo<KIND>::S;
    constexpr int STAGED = Geo<KIND>::STAGED;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64* scount = reinterpret_cast<u64*>(smem_raw);
    u32* sw = reinterpret_cast<u32*>(scount + T);
    u32* bm = sw + STAGED;
    u32* sstart = bm + R * WINW * T;
    u32* slotp = sstart + T;
    u32* tab = slotp + 4;
    u32* sroot = tab + (size_t)a.L * T;

    const u32 tile = claim_tile(a.tile_counter, slotp);
    const int t = threadIdx.x;
    const u64 first_sub = (u64)tile * T;
    const u32 nvalid = (u32)min((u64)T, a.nsub - first_sub);
    const int gk = a.code.k;
    const int L = a.L;

    Src src;
    src.g = a.words;
    src.base = a.base;
    src.total_bits = a.total_bits;
    src.nwords = (a.base + a.total_bits + 31) >> 5;
    src.sm = sw;
    src.sm_w0 = first_sub * (S / 32);
    src.staged = STAGED;
    for (int i = t; i < STAGED; i += T) {
        const u64 k = src.sm_w0 + i;
        sw[i] = k < src.nwords ? __ldg(a.words + k) : 0u;
    }
    Code code = a.code;
    if (KIND == kCodeHuffman) {
        for (int i = t; i < (1 << code.rb); i += T) sroot[i] = __ldg(a.root_global + i);
        code.root = sroot;
    }
    __syncthreads();

    const u64 B = (first_sub + t) * (u64)S;
    const u64 Bend = min(B + S, a.total_bits);

    // ---- 1. transition table of my subsequence ----
    bool done1 = false;
    if (KIND == kCodeGolombRice && gk <= 30) done1 = gr_lockstep_table(src, B, Bend, gk, tab, t, (u32)t < nvalid);
    if ((u32)t < nvalid && !done1) {
        u32 rx[R] = {}, rc[R] = {};
        int nroots = 0;
        auto bmw = [&](int r, int w) -> u32& { return bm[(r * WINW + w) * T + t]; };
        auto popc_below = [&](int r, u32 q) {
            u32 c = 0;
            for (u32 w = 0; w < (q >> 5); ++w) c += __popc(bmw(r, (int)w));
            if (q & 31u) c += __popc(bmw(r, (int)(q >> 5)) & ((1u << (q & 31u)) - 1u));
            return c;
        };
        for (int e = 0; e < L; ++e) {
            const u64 off = entry_offset<KIND>(src, (u32)e, B, gk);
            u64 p = B + off;
            u32 ox = kOOD, oc = 0;
            if (p >= Bend) {  // no codeword starts here: the entry passes through
                ox = Bend == B + S ? entry_index<KIND>(off - S, L, gk) : kOOD;
                tab[e * T + t] = ox;
                continue;
            }
            int hit = -1;
            if (off < (u64)WIN) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (r < nroots && ((bmw(r, (int)(off >> 5)) >> (off & 31u)) & 1u)) hit = r;
            }
            if (hit >= 0) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (r == hit) {
                        ox = rx[r];
                        oc = rc[r];
                    }
                oc -= popc_below(hit, (u32)off);
                tab[e * T + t] = ox | (oc << 8);
                continue;
            }
            const bool rec = nroots < R && off < (u64)WIN;
            if (rec)
                for (int w = 0; w < WINW; ++w) bmw(nroots, w) = 0u;
            int cw = (int)(off >> 5);
            u32 cbits = rec ? (1u << (off & 31u)) : 0u;
            u32 rw[R];
#pragma unroll
            for (int r = 0; r < R; ++r) rw[r] = (r < nroots && off < (u64)WIN) ? bmw(r, cw) : 0u;
            Dec<KIND> d;
            d.init(src, p);
            u32 c = 0;
            bool merged = false;
            while (p < Bend) {
                u64 v;
                p += d.step(src, code, p, v, false);
                ++c;
                if (p < Bend && p - B < (u64)WIN) {
                    const u32 q = (u32)(p - B);
                    const int w = (int)(q >> 5);
                    if (w != cw) {
                        if (rec) bmw(nroots, cw) = cbits;
                        cbits = 0u;
                        cw = w;
#pragma unroll
                        for (int r = 0; r < R; ++r) rw[r] = r < nroots ? bmw(r, w) : 0u;
                    }
                    const u32 bit = 1u << (q & 31u);
                    int h = -1;
                    u32 hx = 0, hc = 0;
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (r < nroots && (rw[r] & bit)) {
                            h = r;
                            hx = rx[r];
                            hc = rc[r];
                        }
                    if (h >= 0) {
                        merged = true;
                        ox = hx;
                        oc = c + hc - popc_below(h, q);
                        break;
                    }
                    cbits |= bit;
                }
            }
            if (!merged) {
                if (rec && cw < WINW) bmw(nroots, cw) = cbits;
                ox = (Bend == B + S && p >= Bend) ? entry_index<KIND>(p - (B + S), L, gk) : kOOD;
                oc = c;
                if (rec) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (r == nroots) {
                            rx[r] = ox;
                            rc[r] = c;
                        }
                    ++nroots;
                }
            }
            tab[e * T + t] = ox | (oc << 8);
        }
    }
    __syncthreads();

    // ---- 2. composed table of the block (warp 0; lane holds entries lane and lane + 32) ----
    // ---- 3. look-back over predecessor blocks ----
    // ---- 4. true entry of every subsequence ----
    if (t < 32) {
        u32 gx[2];
        u64 gc[2];
        for (int h = 0; h < 2; ++h) {
            const int e = t + 32 * h;
            u32 x = e < L ? (u32)e : kOOD;
            u64 c = 0;
            for (u32 j = 0; j < nvalid && x != kOOD; ++j) {
                const u32 v = tab[x * T + j];
                c += v >> 8;
                x = v & 0xffu;
            }
            gx[h] = x;
            gc[h] = c;
        }
        u64 E = 0, C = 0;
        bool failed = false;
        if (tile > 0) {
            for (int h = 0; h < 2; ++h) st_volatile(&a.agg[(u64)tile * kMaxL + t + 32 * h], (u64)gx[h] | (gc[h] << 8));
            __threadfence();
            __syncwarp();
            if (t == 0) st_volatile(&a.flag[tile], 1u);
            // G: composition of the aggregates walked so far (identity to start).
            u32 Gx[2] = {(u32)t, (u32)t + 32};
            u64 Gc[2] = {0, 0};
            long long pidx = (long long)tile - 1;
            u32 spins = 0;
            bool need_pred = false;
            while (true) {
                u32 f = 0;
                if (t == 0) f = ld_volatile(&a.flag[pidx]);
                f = __shfl_sync(kFullMask, f, 0);
                if (f == 0) {
                    if (++spins > kSpinLimit) {
                        failed = true;
                        break;
                    }
                    if (spins > 64) __nanosleep(100);
                    continue;
                }
                __threadfence();
                if (f == 2) {
                    const u64 X = ld_volatile(&a.inc[(u64)pidx * 2]);
                    const u64 CX = ld_volatile(&a.inc[(u64)pidx * 2 + 1]);
                    if (pidx == (long long)tile - 1) {  // exact entry from the direct predecessor
                        E = X;
                        C = CX;
                        break;
                    }
                    const u32 Xi = entry_index<KIND>(X, L, gk);
                    const u32 Xs = Xi == kOOD ? 0u : Xi;
                    const u32 ex0 = __shfl_sync(kFullMask, Gx[0], Xs & 31u), ex1 = __shfl_sync(kFullMask, Gx[1], Xs & 31u);
                    const u64 ec0 = __shfl_sync(kFullMask, Gc[0], Xs & 31u), ec1 = __shfl_sync(kFullMask, Gc[1], Xs & 31u);
                    const u32 gxX = Xs < 32u ? ex0 : ex1;
                    if (Xi == kOOD || gxX == kOOD) {
                        need_pred = true;  // the composition does not cover this entry
                    } else {
                        E = gxX;
                        C = CX + (Xs < 32u ? ec0 : ec1);
                    }
                    break;
                }
                // aggregate F of block pidx: G <- G o F (both halves read G before either is
                // overwritten)
                u32 nx[2];
                u64 nc[2];
                for (int h = 0; h < 2; ++h) {
                    const u64 fv = ld_volatile(&a.agg[(u64)pidx * kMaxL + t + 32 * h]);
                    const u32 y = (u32)(fv & 0xffu);
                    const u32 yy = y == kOOD ? 0u : y;
                    const u32 gx0 = __shfl_sync(kFullMask, Gx[0], yy & 31u), gx1 = __shfl_sync(kFullMask, Gx[1], yy & 31u);
                    const u64 gc0 = __shfl_sync(kFullMask, Gc[0], yy & 31u), gc1 = __shfl_sync(kFullMask, Gc[1], yy & 31u);
                    nx[h] = y == kOOD ? kOOD : (yy < 32u ? gx0 : gx1);
                    nc[h] = (fv >> 8) + (yy < 32u ? gc0 : gc1);
                }
                for (int h = 0; h < 2; ++h) {
                    Gx[h] = (t + 32 * h < L) ? nx[h] : kOOD;
                    Gc[h] = nc[h];
                }
                --pidx;
                if (pidx < 0) {  // cannot happen: tile 0 always publishes its inclusive value
                    failed = true;
                    break;
                }
            }
            if (need_pred && !failed) {
                // wait for the direct predecessor's exact exit
                spins = 0;
                while (true) {
                    u32 f = 0;
                    if (t == 0) f = ld_volatile(&a.flag[tile - 1]);
                    f = __shfl_sync(kFullMask, f, 0);
                    if (f == 2u) break;
                    if (++spins > kSpinLimit) {
                        failed = true;
                        break;
                    }
                    if (spins > 64) __nanosleep(100);
                }
                __threadfence();
                if (!failed) {
                    E = ld_volatile(&a.inc[(u64)(tile - 1) * 2]);
                    C = ld_volatile(&a.inc[(u64)(tile - 1) * 2 + 1]);
                }
            }
        }
        // Fast path: my composed table covers E -> publish my inclusive value right away.
        // (E is an entry index when it came from a composed table, an offset when it came
        // from a predecessor's walk; entry_index maps both.)
        const u32 Ei = entry_index<KIND>(E, L, gk);
        const u32 Es = Ei == kOOD ? 0u : Ei;
        const u32 mx0 = __shfl_sync(kFullMask, gx[0], Es & 31u), mx1 = __shfl_sync(kFullMask, gx[1], Es & 31u);
        const u64 mc0 = __shfl_sync(kFullMask, gc[0], Es & 31u), mc1 = __shfl_sync(kFullMask, gc[1], Es & 31u);
        const u32 tabX = Es < 32u ? mx0 : mx1;
        const bool fast = !failed && Ei != kOOD && tabX != kOOD;
        if (t == 0) {
            if (failed) atomicOr(a.need_fallback, kWaitExpired);
            if (fast) {
                st_volatile(&a.inc[(u64)tile * 2], (u64)tabX);
                st_volatile(&a.inc[(u64)tile * 2 + 1], C + (Es < 32u ? mc0 : mc1));
                __threadfence();
                st_volatile(&a.flag[tile], 2u);
            }
            // walk my subsequences from the true entry (x: offset into subsequence j)
            u64 x = E;
            if (KIND == kCodeGolombRice && E > (u64)gk) x = entry_offset<KIND>(src, (u32)(gk + 1), first_sub * S, gk);
            u64 c = C;
            for (u32 j = 0; j < nvalid; ++j) {
                sstart[j] = (u32)min(x, (u64)0xffffffffu);
                scount[j] = c;
                const u32 xi = entry_index<KIND>(x, L, gk);
                const u32 v = xi != kOOD ? tab[xi * T + j] : kOOD;
                if ((v & 0xffu) != kOOD) {
                    c += v >> 8;
                    x = entry_offset<KIND>(src, v & 0xffu, (first_sub + j + 1) * S, gk);
                } else {
                    const u64 Bj = (first_sub + j) * S;
                    const u64 Ej = min(Bj + S, a.total_bits);
                    u64 pp = Bj + x;
                    if (pp < Ej) {
                        Dec<KIND> d;
                        d.init(src, pp);
                        while (pp < Ej) {
                            u64 val;
                            pp += d.step(src, code, pp, val, false);
                            ++c;
                        }
                    }
                    x = pp >= Bj + S ? pp - (Bj + S) : 0ull;
                }
            }
            if (!fast) {
                st_volatile(&a.inc[(u64)tile * 2], x);
                st_volatile(&a.inc[(u64)tile * 2 + 1], c);
                __threadfence();
                st_volatile(&a.flag[tile], 2u);
            }
            if (tile == gridDim.x - 1) *a.total_codewords = c;
        }
    }
    __syncthreads();

    // ---- 5. decode my subsequence from its true entry ----
    if ((u32)t < nvalid && !(*(volatile u32*)a.need_fallback)) {
        u64 idx = scount[t];
        u64 p = B + sstart[t];
        if (p < Bend && idx < a.nsym) {
            Dec<KIND> d;
            d.init(src, p);
            if (a.out_width == 1) {
                ByteOut bo{static_cast<u8*>(a.out), idx, 0u};
                while (p < Bend && idx < a.nsym) {
                    u64 v;
                    const u64 len = d.step(src, code, p, v, true);
                    if (p + len > a.total_bits) {
                        atomicOr(a.err, kErrBadStream);
                        break;
                    }
                    bo.put(idx, v);
                    ++idx;
                    p += len;
                }
                bo.flush(idx);
            } else {
                while (p < Bend && idx < a.nsym) {
                    u64 v;
                    const u64 len = d.step(src, code, p, v, true);
                    if (p + len > a.total_bits) {
                        atomicOr(a.err, kErrBadStream);
                        break;
                    }
                    if (a.out_width == 4) static_cast<u32*>(a.out)[idx] = (u32)v;
                    else static_cast<u64*>(a.out)[idx] = v;
                    ++idx;
                    p += len;
                }
            }
        }
    }
}

// ------------------------------------------------- self-synchronising decoder ----------
// Decoding from a wrong bit offset falls in step with the right codewords after a few of them
// for nearly every code, so the subsequences (a.S bits, one per thread) are decoded from a
// guess and then corrected: every thread decodes its subsequence from its first bit, takes the
// exit its predecessor arrived at as its entry and decodes again if that differs, until nothing
// changes.  A state in which every entry is the predecessor's exit is the one true decoding
// from the first thread's entry, whatever the guesses were, so the result is exact for any
// prefix code; only the number of rounds depends on the code.
//
// The first G threads of a block redo the last G subsequences of the block before, so that the
// block's own entry has normally fallen in step as well.  A block publishes (entry it assumed,
// exit, codewords); a later block walks back over a chain of blocks whose assumed entries match
// the exits before them, up to one whose result is final (128 at a time), and so gets its true
// entry and its output position.  A block whose assumption was wrong decodes again from the
// true entry.  Waits are bounded.  Streams that do not fall in step in time (kNotConverged, or too many
// wrong assumptions) are left to decode_stream_kernel, whose entry tables do not depend on it.
//
// What bounds it: the dependent chain of codewords within a subsequence (two word reads, a
// funnel shift, a table read), hidden by the other warps.  A subsequence is an odd number of
// words, so that lanes at the same place of theirs read distinct banks.  Measured against the
// entry-table decoder on one B200: the Golomb-Rice stream of 64M terrain points (truncated
// octahedron, L2 0.001; 150 MB in, 256 MB out) 2187 -> 426 us, of 1013 points 119 -> 20 us; the
// Huffman streams of a 120K-point direct container 273 -> 47 us, of 8M points (cube, L2 0.1)
// 568 -> 113 us.
constexpr int kSyncThreads = 128;
constexpr int kSyncHalo = 8;
// When a block gives up, looked at after every fourth round (in every round, 120K points took 2 us longer): a
// quarter of its threads still change after eight, or the rounds took this long (again from the true entry:
// shorter).  Of the streams of all kinds of clouds that fall in step, the slowest takes 39 rounds and 207000
// clocks; half as long turned some of them away, which are then three times slower.  With 64 rounds, all blocks to
// themselves and 256 second decodings, a stream of 16M bits that never falls in step took 0.48 ms more than its
// entry tables alone (now 0.09), of 120K bits 0.5 (0.13), and 7M uniform points, whose symbols have long runs,
// took 2.0-2.2 ms (1.4 when the entry tables came first, now 0.98).
constexpr int kRoundsPerLook = 4;
constexpr u32 kSettleClocks = 220000, kRedoClocks = 60000;
// Blocks that may decode again; each makes all later ones wait, some 20 us.
constexpr u32 kFreeRedos = 2, kBlocksPerRedo = 256;
// Window of the several-symbols table: at least 7 bits (an entry per thread), for codes shorter than that too.
// As narrow as the code, a round of a two-bit code took 15400 clocks; with 7 bits runs of its symbols fall in
// step in 150 us where they took 260 (60K symbols), and 1013 points decompress in 107 us instead of 118.
constexpr int kMinMultiBits = 7, kMaxMultiBits = 10;

struct SyncArgs {
    const u32* words;
    u32 base;
    u64 total_bits;
    u64 nsub;
    int S, G;
    Code code;
    int mb;          // Huffman: window bits of the several-symbols table
    int multi_out;   // its symbols are the values (all below 256)
    u64 nsym;
    int out_width;
    void* out;
    Status* status;  // per tile (tile_state)
    u32* tile_counter;
    u32* err;
    u32* need_fallback;
    u32* redone;
    unsigned long long* total_codewords;
};

__host__ __device__ inline size_t sync_smem(int S, int rb, int mb) {
    return 8 * kSyncThreads + (rb ? (8ull << mb) + (4ull << rb) : 0) + 4 * (size_t)(kSyncThreads * S / 32 + kSyncHalo);
}

// A block's published state (device_common.cuh: Status): lo = the exit relative to the next block's
// first bit << 32 | the assumed entry relative to the block's, hi = codewords (of the block; through
// the block once final) and the flag (1 assumed, 2 final).
__device__ __forceinline__ Pair tile_state(u64 codewords, u64 entry, u64 exit) {
    return Pair{(exit << 32) | entry, codewords};
}

// A thread's run of 32-bit words out[first], out[first + 1], ..: four at a time as one 16-byte
// store where they lie on a 16-byte boundary.  (A lane's stores land in sectors of their own, so
// their number is what the store path is busy with.)
struct WordRun {
    u32* out;
    u64 first;
    u32 a, b, c, d;  // the last four words, d the latest
    __device__ __forceinline__ void put(u64 i, u32 v) {
        a = b;
        b = c;
        c = d;
        d = v;
        if ((i & 3u) == 3u) {
            if (i - 3u >= first && i >= 3u) {
                *reinterpret_cast<uint4*>(out + i - 3u) = make_uint4(a, b, c, d);
            } else {
                rest(i + 1, 3u);
            }
        }
    }
    // the last n (1..3) words before `end`, those from `first` on
    __device__ __forceinline__ void rest(u64 end, u32 n) {
        if (n > 0u && end > first) out[end - 1] = d;
        if (n > 1u && end > first + 1) out[end - 2] = c;
        if (n > 2u && end > first + 2) out[end - 3] = b;
    }
    __device__ __forceinline__ void finish(u64 end) { rest(end, (u32)(end & 3u)); }
};

// A thread's run of bytes from `first` on; whole words go through a WordRun.
struct ByteRun {
    u8* out;
    u64 first, at;
    u64 acc;  // bytes of the word that holds `at`, and up to three beyond
    WordRun w;
    __device__ __forceinline__ void begin(u8* o, u64 i) {
        out = o;
        first = at = i;
        acc = 0;
        w.out = reinterpret_cast<u32*>(o);
        w.first = (i + 3) >> 2;
        w.a = w.b = w.c = w.d = 0;
    }
    __device__ __forceinline__ void bytes(u64 lo, u64 hi, u32 v) const {  // [lo, hi) of one word
        for (u64 j = lo; j < hi; ++j) out[j] = (u8)(v >> ((j & 3u) * 8u));
    }
    // n (1..4) bytes, the first in the low byte
    __device__ __forceinline__ void put(u32 v, u32 n) {
        const u32 k = (u32)at & 3u;
        acc |= (u64)v << (8u * k);
        at += n;
        if (k + n >= 4u) {
            const u64 i = (at - n) >> 2;
            if (i >= w.first) w.put(i, (u32)acc);
            else bytes(first, 4 * i + 4, (u32)acc);
            acc >>= 32;
        }
    }
    __device__ __forceinline__ void finish() {
        const u64 whole = at >> 2;
        if (whole > w.first) w.finish(whole);
        const u64 lo = max(first, whole * 4);
        if (lo < at) bytes(lo, at, (u32)acc);
    }
};

// What a block's threads decode with: the staged words (byte-swapped for MSB-first codes), whose
// bit 0 is stream bit `org`, and the code.  Positions in the staged words are 32-bit (`q`).
template <int KIND>
struct SyncStream {
    const u32* sw;
    u64 org;
    Code code;
    // Huffman, per window of mb bits, the codewords that lie in it: bits taken and number of all of
    // them (bytes 0 and 1; 0: read one codeword) and of the first four (bytes 2 and 3)
    const u32* mlen;
    const u32* msym;  // the symbols of those four
    int mb;
    Src g;  // unstaged, for codewords that do not fit the 32-bit window

    __device__ __forceinline__ u32 window(u32 q) const {
        const u32* w = sw + (q >> 5);
        return KIND == kCodeGolombRice ? __funnelshift_r(w[0], w[1], q) : __funnelshift_l(w[1], w[0], q);
    }
    // One codeword at q: its value and its length, which may exceed 32 bits (Golomb-Rice and
    // exp-Golomb; Huffman: kFar for a prefix that is no code).
    __device__ __forceinline__ u64 one(u32 q, u64& v, bool want) const {
        const u32 win = window(q);
        const int k = code.k;
        if (KIND == kCodeHuffman) {
            u32 sym;
            const u32 len = huff_lookup(code, win, sym);
            v = 0;
            if (!len) return kFar;
            if (want) v = code.symvals ? __ldg(&code.symvals[sym]) : (u64)sym;
            return len;
        }
        if (KIND == kCodeGolombRice) {
            const u32 t = (u32)__ffs((int)~win) - 1u;
            if (t < 32u && k <= 32) {
                if (want) {
                    const u32 r = window(q + t + 1u);
                    v = ((u64)t << k) | (k >= 32 ? r : r & ((1u << k) - 1u));
                }
                return t + 1u + (u32)k;
            }
            return gr_generic(g, org + q, k, v);
        }
        const u32 z = (u32)__clz((int)win);
        if (2u * z + 1u + (u32)k <= 32u) {
            const u32 n1 = (win << z) >> (31u - z);
            const u32 low = k ? __brev((win << (2u * z + 1u)) >> (32 - k)) >> (32 - k) : 0u;
            const u64 u = ((u64)(n1 - 1u) << k) | low;
            v = code.zigzag ? ((u >> 1) ^ (~(u & 1ull) + 1ull)) : u;
            return 2u * z + 1u + (u32)k;
        }
        return eg_generic(g, org + q, k, code.zigzag, v);
    }
    // From q to the first codeword start at or after qe; adds the codewords passed to c.
    __device__ __forceinline__ u64 walk(u32 q, u32 qe, u32& c) const {
        while (q < qe) {
            if (KIND == kCodeHuffman && q + (u32)mb <= qe) {  // every codeword of the window starts before qe
                const u32 e = mlen[window(q) >> (32 - mb)];
                if (e) {
                    q += e & 0xffu;
                    c += (e >> 8) & 0xffu;
                    continue;
                }
            }
            ++c;
            if (KIND == kCodeGolombRice) {
                const u32 t = (u32)__ffs((int)~window(q)) - 1u;
                if (t < 32u) {
                    q += t + 1u + (u32)code.k;
                    continue;
                }
            }
            u64 v;
            const u64 len = one(q, v, false);
            if (len >= kFar) return org + q + len;
            q += (u32)len;
        }
        return org + q;
    }
};

template <int KIND>
__global__ void __launch_bounds__(kSyncThreads) decode_sync_kernel(SyncArgs a) {
    constexpr int TT = kSyncThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ u32 slot, given_up, late;
    __shared__ u64 s_assumed, s_entry, s_first, s_wsum[TT / 32];
    u64* sx = reinterpret_cast<u64*>(smem_raw);
    u32* mlen = reinterpret_cast<u32*>(sx + TT);
    u32* msym = mlen + (KIND == kCodeHuffman ? (1 << a.mb) : 0);
    u32* root = msym + (KIND == kCodeHuffman ? (1 << a.mb) : 0);
    u32* sw = root + (KIND == kCodeHuffman ? (1 << a.code.rb) : 0);

    const u32 tile = claim_tile(a.tile_counter, &slot);
    const int t = threadIdx.x, S = a.S, G = a.G;
    const u32 lane = lane_id();
    const int staged = TT * S / 32 + kSyncHalo;
    const long long sub = (long long)tile * (TT - G) - G + t;  // my subsequence
    const int first_t = tile == 0 ? G : 0;                     // the block's first thread with one
    const bool valid = t >= first_t && sub < (long long)a.nsub;

    SyncStream<KIND> str;
    str.g.g = a.words;
    str.g.base = a.base;
    str.g.total_bits = a.total_bits;
    str.g.nwords = (a.base + a.total_bits + 31) >> 5;
    str.g.sm = nullptr;
    str.g.sm_w0 = 0;
    str.g.staged = 0;
    str.sw = sw;
    str.code = a.code;
    str.mlen = mlen;
    str.msym = msym;
    str.mb = a.mb;
    // (tile 0 stages from the stream's start)
    const u64 w0 = (u64)((long long)tile * (TT - G) - (tile == 0 ? 0 : G)) * (u32)(S / 32);
    str.org = w0 * 32 - a.base;
    const u32 why_not = t == 0 ? ld_volatile(a.need_fallback) : 0u;
#pragma unroll 8
    for (int i = t; i < staged; i += TT) {
        const u64 k = w0 + (u64)i;
        const u32 x = k < str.g.nwords ? __ldg(a.words + k) : 0u;
        sw[i] = KIND == kCodeGolombRice ? x : __byte_perm(x, 0, 0x0123);
    }
    if (t == 0) given_up = why_not & ~kWideValue;
    if (KIND == kCodeHuffman) {
#pragma unroll 8
        for (int i = t; i < (1 << a.code.rb); i += TT) root[i] = __ldg(a.code.root + i);
        str.code.root = root;
        __syncthreads();
        for (int w = t; w < (1 << a.mb); w += TT) {
            u32 at = 0, n = 0, syms = 0, four = 0;
            while (at < (u32)a.mb) {
                const u32 e = root[(((u32)w << (32 - a.mb)) << at) >> (32 - a.code.rb)];
                const u32 len = e >> 24;
                if (len == 0u || len >= 128u || at + len > (u32)a.mb) break;
                at += len;
                if (n < 4) {
                    syms |= (e & 0xffu) << (8 * n);
                    four = at | ((n + 1) << 8);
                }
                ++n;
            }
            mlen[w] = at | (n << 8) | (four << 16);
            msym[w] = syms;
        }
    }
    __syncthreads();
    if (given_up) return;  // (whoever waits for this block looks at need_fallback too)

    const u64 B = valid ? (u64)sub * (u32)S : 0ull;
    const u64 Bend = valid ? min(B + (u64)S, a.total_bits) : 0ull;
    u64 entry = B;
    u32 count = 0;
    // Rounds from thread `from` on (its entry stays) until every entry is the exit before it.
    auto settle = [&](int from, bool active, u32 clocks) {
        const u32 begin = (u32)clock();
        for (int round = 0;; ++round) {
            if (active) {
                count = 0;
                sx[t] = entry < Bend ? str.walk((u32)(entry - str.org), (u32)(Bend - str.org), count) : entry;
            }
            __syncthreads();
            const u64 e = t > from && valid ? sx[t - 1] : entry;
            active = valid && t > from && e != entry;
            entry = e;
            if (!__syncthreads_or(active)) return true;
            if (round % kRoundsPerLook == kRoundsPerLook - 1) {
                if (t == 0) late = (u32)clock() - begin > clocks;
                if ((__syncthreads_count(active) > TT / 4 && round > kRoundsPerLook) || late) return false;
            }
        }
    };
    bool settled = settle(first_t, valid, kSettleClocks);

    // codewords before mine within the block's own subsequences, and the block's total
    const bool own = valid && t >= G;
    u64 before = 0, total = 0;
    auto sum_counts = [&]() {
        const u32 mine = own ? count : 0u;
        const u32 incl = warp_incl_add(mine);
        __syncthreads();  // (s_wsum may still be read by the previous call's)
        if (lane == 31) s_wsum[t >> 5] = incl;
        __syncthreads();
        u64 b = incl - mine, all = 0;
        for (int w = 0; w < TT / 32; ++w) {
            if (w < (t >> 5)) b += s_wsum[w];
            all += s_wsum[w];
        }
        before = b;
        total = all;
    };
    sum_counts();
    const int last_t = (int)min((long long)TT - 1, (long long)a.nsub - 1 - ((long long)tile * (TT - G) - G));
    if (t == G) s_assumed = entry;
    __syncthreads();
    const u64 assumed = s_assumed;  // (read by slower warps while warp 0 already writes s_entry)

    // first bit of this block's own subsequences and of the next block's
    const u64 tile_at = (u64)tile * (u64)(TT - G) * (u64)S, next_at = tile_at + (u64)(TT - G) * (u64)S;
    auto exit_of = [&]() { return sx[last_t] > next_at ? sx[last_t] - next_at : 0ull; };  // (0: the last block)
    if (t < 32) {
        bool failed = !settled || (exit_of() >> 32) != 0 || ((assumed - tile_at) >> 32) != 0;
        u32 why = kNotConverged;
        u64 E = assumed - tile_at, C = 0;
        if (tile > 0) {
            if (lane == 0 && !failed) st_status(&a.status[tile], tile_state(total, assumed - tile_at, exit_of()), 1u);
            // 128 blocks per step, four per lane (the nearest first)
            long long top = (long long)tile - 1;
            u64 pend = 0;
            u32 spins = 0;
            while (!failed) {
                u32 f[4];
                u64 n[4], ex[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const long long q = top - 4 * (long long)lane - j;
                    f[j] = 2u;
                    Pair v{0, 0};
                    if (q >= 0) v = ld_status(&a.status[q], f[j]);
                    n[j] = v.hi;
                    ex[j] = v.lo;
                }
                // my four up to my first final one, chained to the next lane's first exit
                const u64 xnext = __shfl_down_sync(kFullMask, ex[0] >> 32, 1);
                bool bad = false, fin = false;
                u64 add = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (fin) continue;
                    add += n[j];
                    if (f[j] == 2u) {
                        fin = true;
                    } else if (f[j] == 0u) {
                        bad = true;
                    } else {
                        const u64 x = j < 3 ? ex[j < 3 ? j + 1 : 3] >> 32 : xnext;
                        if ((j < 3 || lane < 31u) && (ex[j] & 0xffffffffull) != x) bad = true;
                    }
                }
                const u32 fm = __ballot_sync(kFullMask, fin);
                const u32 last = fm ? (u32)__ffs(fm) - 1u : 31u;
                const u64 x0 = __shfl_sync(kFullMask, ex[0] >> 32, 0);
                const bool link = top == (long long)tile - 1 || pend == x0;
                if (__any_sync(kFullMask, bad && lane <= last) || !link) {
                    const u32 given_up = __shfl_sync(kFullMask, lane == 0 ? ld_volatile(a.need_fallback) : 0u, 0);
                    if (++spins > kSpinLimit) {
                        failed = true;
                        why = kWaitExpired;
                    } else if ((given_up & ~kWideValue) != 0u) {
                        failed = true;
                    }
                    if (spins > 64) __nanosleep(100);
                    if (!link) {  // the chain's last link has been decoded again: start over
                        top = (long long)tile - 1;
                        C = 0;
                    }
                    continue;
                }
                if (top == (long long)tile - 1) E = x0;
                C += warp_sum(lane <= last ? add : 0ull);
                if (fm) break;
                pend = __shfl_sync(kFullMask, ex[3] & 0xffffffffull, 31);
                top -= 128;
            }
        }
        if (lane == 0) {
            if (failed) {  // seen by whoever reads the status below
                atomicOr(a.need_fallback, why);
                __threadfence();
            }
            const bool same = E == assumed - tile_at;
            if (!failed && !same && atomicAdd(a.redone, 1u) >= kFreeRedos + gridDim.x / kBlocksPerRedo) atomicOr(a.need_fallback, kNotConverged);
            if (failed || same) st_status(&a.status[tile], tile_state(C + total, 0ull, exit_of() & 0xffffffffull), 2u);
            s_entry = failed ? assumed : tile_at + E;
            s_first = C;
        }
    }
    __syncthreads();
    if (s_entry != assumed) {  // block-uniform: decode again from the true entry
        if (t == G) entry = s_entry;
        const bool ok = settle(G, t == G, kRedoClocks);
        sum_counts();
        if (t == 0) {
            if (!ok || (exit_of() >> 32) != 0) {
                atomicOr(a.need_fallback, kNotConverged);
                __threadfence();
            }
            st_status(&a.status[tile], tile_state(s_first + total, 0ull, exit_of() & 0xffffffffull), 2u);
        }
    }
    if (tile == gridDim.x - 1 && t == 0) *a.total_codewords = s_first + total;

    u64 idx = s_first + before;
    if (own && entry < Bend && idx < a.nsym && !(ld_volatile(a.need_fallback) & ~kWideValue)) {
        u32 q = (u32)(entry - str.org);
        const u32 qe = (u32)(Bend - str.org);
        const bool bytes = a.out_width == 1;
        ByteRun br;
        br.begin(static_cast<u8*>(a.out), idx);
        WordRun wr{static_cast<u32*>(a.out), idx, 0, 0, 0, 0};
        bool wide = false;
        while (q < qe && idx < a.nsym) {
            if (KIND == kCodeHuffman && a.multi_out && q + (u32)a.mb <= qe && idx + 4 <= a.nsym) {
                const u32 w = str.window(q) >> (32 - a.mb);
                const u32 e = mlen[w] >> 16;
                if (e) {
                    u32 syms = msym[w];
                    const u32 n = e >> 8;
                    q += e & 0xffu;
                    if (bytes) {
                        br.put(syms, n);
                        idx += n;
                    } else {
                        for (u32 i = 0; i < n; ++i, syms >>= 8, ++idx) wr.put(idx, syms & 0xffu);
                    }
                    continue;
                }
            }
            u64 v;
            const u64 len = str.one(q, v, true);
            if (str.org + q + len > a.total_bits) {
                atomicOr(a.err, kErrBadStream);
                break;
            }
            if (KIND == kCodeHuffman && bytes) {
                br.put((u32)v & 0xffu, 1u);
            } else if (a.out_width == 4) {
                wr.put(idx, (u32)v);
                wide |= (v >> 32) != 0;
            } else {
                static_cast<u64*>(a.out)[idx] = v;
            }
            ++idx;
            if (len >= kFar) break;  // past every subsequence of this thread
            q += (u32)len;
        }
        if (KIND == kCodeHuffman && bytes) br.finish();
        else if (a.out_width == 4 && idx > wr.first) wr.finish(idx);
        if (KIND == kCodeGolombRice && wide) atomicOr(a.need_fallback, kWideValue);
    }
}

// One-thread decoder, run by the host after a bounded wait of the parallel decoder expired.
template <int KIND>
__global__ void decode_sequential_kernel(Args a) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    Src src;
    src.g = a.words;
    src.base = a.base;
    src.total_bits = a.total_bits;
    src.nwords = (a.base + a.total_bits + 31) >> 5;
    src.sm = nullptr;
    src.sm_w0 = 0;
    src.staged = 0;  // nothing staged
    Code code = a.code;
    code.root = a.root_global;
    u64 p = 0, i = 0;
    Dec<KIND> d;
    d.init(src, 0);
    while (i < a.nsym && p < a.total_bits) {
        u64 v;
        const u64 len = d.step(src, code, p, v, true);
        if (p + len > a.total_bits) {
            atomicOr(a.err, kErrBadStream);
            break;
        }
        if (a.out_width == 1) static_cast<u8*>(a.out)[i] = (u8)v;
        else if (a.out_width == 4) static_cast<u32*>(a.out)[i] = (u32)v;
        else static_cast<u64*>(a.out)[i] = v;
        ++i;
        p += len;
    }
    *a.total_codewords = i;
}

// A Huffman stream whose codewords all have one length `len` (<= kMaxRootBits): symbol i is
// bits [i len, (i + 1) len) of the stream, one table lookup each, so the stream needs neither entry
// tables nor look-back.  A thread decodes 16 symbols, from one 64-bit window (SHORT: len <= 4) or from
// one per four symbols, through a table of values in shared memory, and stores them in 16-byte pieces.
// Bound by instructions: four symbols per thread through the global table took 64 per symbol; the three
// Huffman streams of 64M terrain points (two of them of one length) took 427 us, with this 262.  A chunk
// that is no codeword sets kErrBadStream, as the chained decoder does.
template <bool SHORT, int WIDTH>
__global__ void __launch_bounds__(256) decode_fixed_kernel(const u32* __restrict__ words, u32 base, u64 nwords,
                                                           int len, const u32* __restrict__ root,
                                                           const u64* __restrict__ symvals, u64 nsym,
                                                           void* out, bool aligned, u32* err) {
    __shared__ uint2 tab[1 << kMaxRootBits];  // value, and whether no codeword
    for (u32 i = threadIdx.x; i < 1u << len; i += blockDim.x) {
        const u32 e = __ldg(root + i), v = e & 0xffffffu;
        tab[i] = make_uint2(symvals ? (u32)__ldg(symvals + v) : v, (e >> 24) != (u32)len);
    }
    __syncthreads();
    constexpr int kPer = SHORT ? 16 : 4;
    auto wbe = [&](u64 k) -> u32 {
        const u32 w = __byte_perm(__ldg(words + (k < nwords ? k : nwords - 1)), 0, 0x0123);
        return k < nwords ? w : 0u;
    };
    const u64 groups = (nsym + 15) / 16;
    for (u64 g = (u64)blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += (u64)gridDim.x * blockDim.x) {
        const u32 cnt = (u32)min((u64)16, nsym - 16 * g);
        u32 v[16], bad = 0;
#pragma unroll
        for (int p = 0; p < 16; p += kPer) {
            const u64 q = (u64)base + (16 * g + p) * (u64)len, k = q >> 5;
            const u32 o = (u32)q & 31u, w0 = wbe(k), w1 = wbe(k + 1), w2 = wbe(k + 2);
            u32 hi = __funnelshift_l(w1, w0, o), lo = __funnelshift_l(w2, w1, o);
#pragma unroll
            for (int j = p; j < p + kPer; ++j) {
                const uint2 e = tab[hi >> (32 - len)];
                hi = __funnelshift_l(lo, hi, len);
                lo <<= len;
                v[j] = e.x;
                bad |= (u32)j < cnt ? e.y : 0u;
            }
        }
        if (WIDTH == 1) {
            u32 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                w[j] = __byte_perm(__byte_perm(v[4 * j], v[4 * j + 1], 0x0040), __byte_perm(v[4 * j + 2], v[4 * j + 3], 0x0040), 0x5410);
            u8* o8 = static_cast<u8*>(out) + 16 * g;
            if (cnt == 16u && aligned) {
                *reinterpret_cast<uint4*>(o8) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
#pragma unroll
                for (u32 j = 0; j < 16; ++j)
                    if (j < cnt) o8[j] = (u8)v[j];
            }
        } else {
            u32* o32 = static_cast<u32*>(out) + 16 * g;
            if (cnt == 16u && aligned) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) *reinterpret_cast<uint4*>(o32 + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            } else {
#pragma unroll
                for (u32 j = 0; j < 16; ++j)
                    if (j < cnt) o32[j] = v[j];
            }
        }
        if (bad) atomicOr(err, kErrBadStream);
    }
}

__global__ void flag_error_kernel(u32* err) { atomicOr(err, kErrBadStream); }
void atomic_flag_host_error(u32* err, cudaStream_t st) { flag_error_kernel<<<1, 1, 0, st>>>(err); }

Args make_args(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits, const DecodeTable& t, int L,
               uint64_t nsym, int out_width, void* out) {
    Args a{};
    a.words = words;
    a.base = (u32)base_bits;
    a.total_bits = total_bits;
    const u64 S = kind == kCodeGolombRice ? (u64)kDecodeSubBitsGR : (u64)kDecodeSubBits;
    a.nsub = (total_bits + S - 1) / S;
    a.L = kind == kCodeGolombRice ? (t.param + 2 < kMaxL ? t.param + 2 : kMaxL) : (L < 1 ? 1 : (L > kMaxL ? kMaxL : L));
    a.code.root = t.root;
    a.code.tree = t.tree;
    a.code.symvals = t.symvals;
    a.code.rb = kind == kCodeHuffman ? t.root_bits : 0;
    a.code.k = t.param;
    a.code.zigzag = t.zigzag;
    a.root_global = t.root;
    a.nsym = nsym;
    a.out_width = out_width;
    a.out = out;
    return a;
}

}  // namespace

void launch_decode_stream(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits, DecodeTable t,
                          int L, uint64_t nsym, int out_width, void* out, uint32_t* flag,
                          unsigned long long* agg, unsigned long long* inc, uint32_t* tile_counter, uint32_t* err,
                          uint32_t* need_fallback, unsigned long long* total_codewords, cudaStream_t st) {
    if (kind == kCodeHuffman && (t.root_bits < 1 || t.root_bits > kMaxRootBits)) {
        atomic_flag_host_error(err, st);  // the host builds tables with 1 <= root_bits <= 11
        return;
    }
    Args a = make_args(kind, words, base_bits, total_bits, t, L, nsym, out_width, out);
    a.flag = flag;
    a.agg = agg;
    a.inc = inc;
    a.tile_counter = tile_counter;
    a.err = err;
    a.need_fallback = need_fallback;
    a.total_codewords = total_codewords;
    const unsigned tiles = (unsigned)((a.nsub + T - 1) / T);
    if (!tiles) return;
    // The launch uses what this stream needs; the function's limit is always set to the
    // largest size any stream can need (the same value from every thread, so concurrent
    // launches from other contexts cannot lower it between this call and the launch).
    const int smem = kind == kCodeGolombRice ? (int)smem_for<kCodeGolombRice>(a.L, a.code.rb)
                                             : (int)smem_for<kCodeHuffman>(a.L, a.code.rb);
    const int smem_max = kind == kCodeGolombRice ? (int)smem_for<kCodeGolombRice>(kMaxL, kMaxRootBits)
                                                 : (int)smem_for<kCodeHuffman>(kMaxL, kMaxRootBits);
    if (kind == kCodeHuffman) {
        cudaFuncSetAttribute(decode_stream_kernel<kCodeHuffman>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        decode_stream_kernel<kCodeHuffman><<<tiles, T, smem, st>>>(a);
    } else if (kind == kCodeGolombRice) {
        cudaFuncSetAttribute(decode_stream_kernel<kCodeGolombRice>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem_max);
        decode_stream_kernel<kCodeGolombRice><<<tiles, T, smem, st>>>(a);
    } else {
        cudaFuncSetAttribute(decode_stream_kernel<kCodeExpGolomb>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem_max);
        decode_stream_kernel<kCodeExpGolomb><<<tiles, T, smem, st>>>(a);
    }
}

SyncGeometry sync_geometry(int kind, uint64_t total_bits) {
    SyncGeometry g{};
    // Subsequences of 33 (Golomb-Rice), 17, 9 or 5 words: the longest that still leaves every SM
    // a few blocks (a round costs a subsequence's whole chain, so short ones settle sooner; long
    // ones need fewer rounds, and fewer of them are decoded twice by neighbouring blocks).
    const uint64_t want = 112ull * 148 * 4;
    int w = kind == kCodeGolombRice ? 33 : 17;
    const int smallest = kind == kCodeGolombRice ? 9 : 5;
    while (w > smallest && total_bits < want * 32 * (uint64_t)w) w = w / 2 + 1;
    g.S = 32 * w;
    const uint64_t nsub = (total_bits + g.S - 1) / g.S;
    if (nsub <= (uint64_t)kSyncThreads) {
        g.tiles = nsub ? 1 : 0;
        return g;
    }
    // decoded ahead of a block: 8192 bits (Golomb-Rice codewords are longer) or 2048
    g.G = (kind == kCodeGolombRice ? 8192 : 2048) / g.S;
    if (g.G < 8) g.G = 8;
    if (g.G > kSyncThreads / 2) g.G = kSyncThreads / 2;
    g.tiles = (nsub + (kSyncThreads - g.G) - 1) / (kSyncThreads - g.G);
    return g;
}

void launch_decode_sync(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits, DecodeTable t,
                        bool byte_symbols, uint64_t nsym, int out_width, void* out, void* status,
                        uint32_t* tile_counter, uint32_t* err, uint32_t* need_fallback, uint32_t* redone, unsigned long long* total_codewords,
                        cudaStream_t st) {
    if (kind == kCodeHuffman && (t.root_bits < 1 || t.root_bits > kMaxRootBits)) {
        atomic_flag_host_error(err, st);  // the host builds tables with 1 <= root_bits <= 11
        return;
    }
    const SyncGeometry g = sync_geometry(kind, total_bits);
    if (!g.tiles) return;
    SyncArgs a{};
    a.words = words;
    a.base = (u32)base_bits;
    a.total_bits = total_bits;
    a.S = g.S;
    a.G = g.G;
    a.nsub = (total_bits + g.S - 1) / g.S;
    a.code.root = t.root;
    a.code.tree = t.tree;
    a.code.symvals = t.symvals;
    a.code.rb = kind == kCodeHuffman ? t.root_bits : 0;
    a.code.k = t.param;
    a.code.zigzag = t.zigzag;
    a.mb = t.root_bits < kMinMultiBits ? kMinMultiBits : t.root_bits < kMaxMultiBits ? t.root_bits : kMaxMultiBits;
    a.multi_out = byte_symbols && !t.symvals;
    a.nsym = nsym;
    a.out_width = out_width;
    a.out = out;
    a.status = static_cast<Status*>(status);
    a.tile_counter = tile_counter;
    a.err = err;
    a.need_fallback = need_fallback;
    a.redone = redone;
    a.total_codewords = total_codewords;
    const unsigned tiles = (unsigned)g.tiles;
    // at most 16.5 KB of words, 16 KB of tables and 1 KB of exits: below the 48 KB that need no opt-in
    const int smem = (int)sync_smem(g.S, a.code.rb, a.mb);
    if (kind == kCodeHuffman)
        decode_sync_kernel<kCodeHuffman><<<tiles, kSyncThreads, smem, st>>>(a);
    else if (kind == kCodeGolombRice)
        decode_sync_kernel<kCodeGolombRice><<<tiles, kSyncThreads, smem, st>>>(a);
    else
        decode_sync_kernel<kCodeExpGolomb><<<tiles, kSyncThreads, smem, st>>>(a);
}

void launch_decode_fixed(const uint32_t* words, uint64_t base_bits, uint64_t total_bits, DecodeTable t, int len,
                         uint64_t nsym, int out_width, void* out, uint32_t* err, cudaStream_t st) {
    if (!nsym) return;
    if (len < 1 || len > kMaxRootBits || len != t.root_bits || (out_width != 1 && out_width != 4) ||
        nsym * (uint64_t)len > total_bits) {
        atomic_flag_host_error(err, st);  // the host only routes complete fixed-length streams here
        return;
    }
    const u64 nwords = (base_bits + total_bits + 31) / 32;
    const u64 threads = (nsym + 15) / 16, want = (threads + 255) / 256;
    const unsigned blocks = (unsigned)(want < 148 * 8 ? want : 148 * 8);
    const bool aligned = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    auto k = out_width == 1 ? (len <= 4 ? decode_fixed_kernel<true, 1> : decode_fixed_kernel<false, 1>)
                            : (len <= 4 ? decode_fixed_kernel<true, 4> : decode_fixed_kernel<false, 4>);
    k<<<blocks, 256, 0, st>>>(words, (u32)base_bits, nwords, len, t.root, t.symvals, nsym, out, aligned, err);
}

void launch_decode_sequential(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits,
                              DecodeTable t, uint64_t nsym, int out_width, void* out,
                              unsigned long long* total_codewords, uint32_t* err, cudaStream_t st) {
    Args a = make_args(kind, words, base_bits, total_bits, t, kMaxL, nsym, out_width, out);
    a.err = err;
    a.total_codewords = total_codewords;
    if (kind == kCodeHuffman)
        decode_sequential_kernel<kCodeHuffman><<<1, 32, 0, st>>>(a);
    else if (kind == kCodeGolombRice)
        decode_sequential_kernel<kCodeGolombRice><<<1, 32, 0, st>>>(a);
    else
        decode_sequential_kernel<kCodeExpGolomb><<<1, 32, 0, st>>>(a);
}

}  // namespace dev
}  // namespace xnyz
