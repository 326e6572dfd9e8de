// Zstandard frame decoder (RFC 8878) usable from host and device code, for the zstd level-3
// frames that wrap the containers (composer/utils.hpp:11-53 writes them with libzstd).
// Decoding is deterministic, so any correct decoder returns libzstd's bytes.
//
// Supported: single zstd frames without dictionary, raw / RLE / compressed blocks, raw / RLE /
// Huffman (1 or 4 streams, tree or repeated tree) literals, predefined / RLE / FSE / repeated
// sequence tables, repeat offsets, an optional content checksum (skipped, not verified).
//
// A Team is the set of threads that decode one frame together: on the GPU a block of 128
// (BlockTeam), on the host one (SoloTeam).  Each Huffman stream is cut into a piece per thread
// (huf_streams_team); FSE tables are built by a thread per symbol; thread 0 walks the sequences'
// states, 64 at a time, and then every thread finds the sources of eight bytes of their output at once.
// A barrier separates each batch of stores from the reads that follow; every branch around a
// barrier depends only on values that all threads hold alike.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define ZD_HD __host__ __device__ __forceinline__
#else
#define ZD_HD inline
#endif

namespace xnyz {
namespace zd {

using u8 = uint8_t;
using u16 = uint16_t;
using u32 = uint32_t;
using u64 = unsigned long long;
using i64 = long long;

enum : int {
    kOk = 0,
    kErrFormat = -1,     // not a frame this decoder handles, or a corrupt one
    kErrDstSize = -2,    // output larger than the destination
    kErrTruncated = -3,  // input ends early
};

constexpr int kMaxBlock = 128 * 1024;
constexpr int kHufMaxBits = 11;

constexpr int kBatch = 64;           // sequences read at once (64 at most)
constexpr int kBatchWords = (kBatch * 89 + 64 + 31) / 32 + 2;     // their bits (89 at most each), the window below and a part word
constexpr u32 kChunkBytes = 2048;    // output of those that are executed at once, if more than one
constexpr int kTeamMax = 128;
// Workspace of one decoder.  On the GPU the tables are in shared memory and `lit` points to the literal
// buffer in global memory.
struct FseEntry {
    u16 base;  // next-state baseline
    u8 sym;
    u8 nb;     // bits to read
};
struct Tables {
    u16 huf[1 << kHufMaxBits];  // (symbol << 8) | bits
    // literal lengths, offsets, match lengths: the code's baseline, and next-state baseline | state bits <<
    // 16 | extra bits << 24
    u32 seq_value[3][512], seq_next[3][512];
    // scratch of the table readers
    short norm[3][256];
    u8 state_sym[3][512];
    FseEntry weights[64];
    u16 next[256];
    u8 w[256], sorted[256];
    u32 count[16];
    int nsym[3], log[3], built[3];
    // of huf_streams_team
    i64 end[kTeamMax];
    u32 num[kTeamMax];
    // a batch of sequences: its bits; where each starts in them and its states; its baselines and extra bits
    // added up; first output byte and first literal (from the batch's); the offset
    u32 q_words[kBatchWords + 2], q_pos;
    u64 q_at[kBatch];
    // literals | all bytes << 32 up to and with each; what becomes of the three last offsets (RepMap)
    u64 q_len[2][kBatch], q_rep[2][kBatch][3];
    u32 q_ll[kBatch], q_off[kBatch], q_start[kBatch + 1], q_lit[kBatch + 1];
    u32 state[3], rep[3];
    // a chunk's bytes: the values of those from outside, and the byte of the chunk that each repeats (or itself)
    u64 q_value[kChunkBytes / 8 + 2];
    alignas(8) u16 q_from[kChunkBytes + 16];
    int msg[4];
};
struct Workspace : Tables {
    u8 lit[kMaxBlock + 32];
};
// Table sizes of the frame so far, held by each thread of the team.
struct Logs {
    int huf_bits = 0;                      // 0: no Huffman table yet
    int seq[3] = {-1, -1, -1};             // -1: no sequence table yet
};

// One host thread.
struct SoloTeam {
    int rank = 0;
    static constexpr int size = 1;
    void sync() const {}
    int min(int v) const { return v; }
};

#ifdef __CUDACC__
// Its first warp and the others, which can work apart for a while.
struct HeadTeam {
    int rank;
    static constexpr int size = 32;
    __device__ __forceinline__ void sync() const { __syncwarp(); }
};
struct TailTeam {
    int rank;
    static constexpr int size = 96;
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync 1, 96;" ::: "memory"); }
};
// A block of 128 threads.
struct BlockTeam {
    int rank;
    int* slot;  // shared
    static constexpr int size = 128;
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ int min(int v) const {
        __syncthreads();
        if (rank == 0) *slot = 0x7fffffff;
        __syncthreads();
        atomicMin(slot, v);
        __syncthreads();
        return *slot;
    }
};
#endif

// ---- little-endian reads ----
ZD_HD u32 rd16(const u8* p) { return (u32)p[0] | ((u32)p[1] << 8); }
ZD_HD u32 rd24(const u8* p) { return (u32)p[0] | ((u32)p[1] << 8) | ((u32)p[2] << 16); }
ZD_HD u32 rd32(const u8* p) { return rd16(p) | (rd16(p + 2) << 16); }
ZD_HD int highbit(u32 v) {
#ifdef __CUDA_ARCH__
    return 31 - __clz((int)v);
#endif
    int n = -1;
    while (v) {
        v >>= 1;
        ++n;
    }
    return n;
}

// Backward bit stream (FSE / Huffman payloads): bits are consumed from the end of the
// buffer towards its start; the last byte's highest set bit marks the end of the padding.
struct BackBits {
    const u8* buf;
    i64 len;    // bytes
    i64 pos;    // bits not yet consumed (from bit 0 of buf)
    i64 total;  // bits after the padding
    i64 wb;     // first byte of the cached 8-byte window
    u64 win;    // buf[wb .. wb+8), bytes outside the buffer as zero
    ZD_HD bool init(const u8* b, u64 n) {
        buf = b;
        len = (i64)n;
        wb = -(1ll << 40);
        if (!n || !b[n - 1]) return false;
        total = (i64)n * 8 - 8 + highbit(b[n - 1]);
        pos = total;
        return true;
    }
    // n <= 32 bits, most significant first; bits before the start read as zero
    ZD_HD u32 read(int n) {
        if (n == 0) return 0;
        pos -= n;
        return peek_at(pos, n);
    }
    ZD_HD u32 peek(int n) { return n ? peek_at(pos - n, n) : 0; }
    // The bits [p, p+n) need bytes p/8 .. p/8+4; the window is refilled 3 bytes below p/8,
    // so the reads that follow (towards the start) hit it for about 32 bits.
    ZD_HD u32 peek_at(i64 p, int n) {
        const i64 byte0 = p >> 3;  // arithmetic shift: negative positions round down
        if (byte0 < wb || byte0 > wb + 3) {
            wb = byte0 - 3;
            {
                u64 v = 0;
                for (int k = 0; k < 8; ++k) {
                    const i64 b = wb + k;
                    const u64 x = buf[b < 0 ? 0 : b < len ? b : len - 1];
                    v |= (b >= 0 && b < len ? x : 0) << (8 * k);
                }
                win = v;
            }
        }
        const int sh = (int)(p - wb * 8);
        return (u32)((win >> sh) & ((1ull << n) - 1));
    }
    ZD_HD bool overflow() const { return pos < 0; }
};

// ---- FSE ----
// Reads a normalized distribution (RFC 8878 4.1.1); returns bytes used or < 0.
ZD_HD int read_ncount(const u8* src, u64 len, int max_log, int max_sym, short* norm, int& nsym, int& log) {
    if (len < 1) return kErrTruncated;
    i64 bitpos = 0;
    auto bits = [&](int n) -> u32 {
        u32 v = 0;  // n <= 10: three bytes
        for (int k = 0; k < 3; ++k) {
            const i64 b = (bitpos >> 3) + k;
            v |= (b < (i64)len ? (u32)src[b] : 0u) << (8 * k);
        }
        return (v >> (bitpos & 7)) & ((1u << n) - 1u);
    };
    log = (int)bits(4) + 5;
    bitpos += 4;
    if (log > max_log) return kErrFormat;
    int remaining = (1 << log) + 1;
    int threshold = 1 << log;
    int nb = log + 1;
    int s = 0;
    bool prev0 = false;
    while (remaining > 1 && s <= max_sym) {
        if (prev0) {
            // repeat flags: 2 bits each, 3 means "3 more and another flag"
            int n0 = s;
            for (;;) {
                const u32 f = bits(2);
                bitpos += 2;
                n0 += (int)f;
                if (f != 3) break;
            }
            if (n0 > max_sym + 1) return kErrFormat;
            while (s < n0) norm[s++] = 0;
            if (s > max_sym) break;
        }
        const int max = (2 * threshold - 1) - remaining;
        int count;
        const u32 low = bits(nb - 1);
        if ((int)low < max) {
            count = (int)low;
            bitpos += nb - 1;
        } else {
            u32 v = bits(nb);
            if ((int)v >= threshold) v -= max;
            count = (int)v;
            bitpos += nb;
        }
        count--;  // -1: "less than 1"
        remaining -= count < 0 ? -count : count;
        norm[s++] = (short)count;
        prev0 = count == 0;
        while (remaining < threshold) {
            nb--;
            threshold >>= 1;
        }
    }
    if (remaining != 1 || s > max_sym + 1) return kErrFormat;
    nsym = s;
    for (int k = s; k <= max_sym; ++k) norm[k] = 0;
    if (bitpos > (i64)len * 8) return kErrTruncated;
    return (int)((bitpos + 7) >> 3);
}

// Decoding table from a normalized distribution (RFC 8878 4.1.1).
ZD_HD int build_fse(const short* norm, int nsym, int log, FseEntry* t, u16* next) {
    const int size = 1 << log;
    int high = size - 1;
    for (int s = 0; s < nsym; ++s) {
        if (norm[s] == -1) {
            t[high--].sym = (u8)s;
            next[s] = 1;
        } else {
            next[s] = (u16)norm[s];
        }
    }
    const int step = (size >> 1) + (size >> 3) + 3, mask = size - 1;
    int p = 0;
    for (int s = 0; s < nsym; ++s) {
        for (int i = 0; i < norm[s]; ++i) {
            t[p].sym = (u8)s;
            do {
                p = (p + step) & mask;
            } while (p > high);
        }
    }
    if (p != 0) return kErrFormat;
    for (int i = 0; i < size; ++i) {
        const int s = t[i].sym;
        const u32 ns = next[s]++;
        const int nb = log - highbit(ns);
        t[i].nb = (u8)nb;
        t[i].base = (u16)((ns << nb) - size);
    }
    return kOk;
}

// Predefined distributions (RFC 8878 3.1.1.3.2.2).
ZD_HD void default_ll(short* n) {
    const short d[36] = {4, 3, 2, 2, 2, 2, 2, 2, 2, 2, 2, 2, 2, 1, 1, 1, 2, 2,
                         2, 2, 2, 2, 2, 2, 2, 3, 2, 1, 1, 1, 1, 1, -1, -1, -1, -1};
    for (int i = 0; i < 36; ++i) n[i] = d[i];
}
ZD_HD void default_ml(short* n) {
    const short d[53] = {1, 4, 3, 2, 2, 2, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
                         1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1, -1, -1};
    for (int i = 0; i < 53; ++i) n[i] = d[i];
}
ZD_HD void default_of(short* n) {
    const short d[29] = {1, 1, 1, 1, 1, 1, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1};
    for (int i = 0; i < 29; ++i) n[i] = d[i];
}

// Literal / match length codes: baseline and extra bits (RFC 8878 3.1.1.3.2.1.1).
ZD_HD void ll_code(int c, u32& base, int& bits) {
    const u32 b[36] = {0,  1,  2,  3,  4,  5,  6,  7,  8,   9,   10,  11,   12,   13,   14,   15,    16,    18,
                       20, 22, 24, 28, 32, 40, 48, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 16384, 32768, 65536};
    const u8 n[36] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 2, 2, 3, 3, 4, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16};
    base = b[c];
    bits = n[c];
}
ZD_HD void ml_code(int c, u32& base, int& bits) {
    if (c < 32) {
        base = (u32)c + 3;
        bits = 0;
        return;
    }
    const u32 b[21] = {35, 37, 39, 41, 43, 47, 51, 59, 67, 83, 99, 131, 259, 515, 1027, 2051, 4099, 8195, 16387, 32771, 65539};
    const u8 n[21] = {1, 1, 1, 1, 2, 2, 3, 3, 4, 4, 5, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16};
    base = b[c - 32];
    bits = n[c - 32];
}

// A bit stream's bits as a thread walks them down: 32-bit words on 4-byte boundaries.  Bits before the
// stream's start read as zero.  (Loads with an index out of range are clamped, not skipped.)
struct Words {
    const u8* base;  // the 4-byte boundary at or before the stream
    u32 skip;        // bits from there to the stream's start
    i64 words;       // words that hold bits of the stream
#ifndef __CUDA_ARCH__
    i64 end;         // bytes from base to the stream's end
#endif
    ZD_HD void open(const u8* src, u64 len) {
        const u32 off = (u32)((u64)src & 3u);
        base = src - off;
        skip = 8u * off;
        words = (i64)((len + off + 3) / 4);
#ifndef __CUDA_ARCH__
        end = (i64)(len + off);
#endif
    }
    ZD_HD u32 word(i64 i) const {
#ifdef __CUDA_ARCH__
        u32 v = reinterpret_cast<const u32*>(base)[i < 0 ? 0 : i < words ? i : words - 1];
        if (i < 0 || i >= words) v = 0;
#else
        u32 v = 0;  // (bytes outside the stream are not touched)
        for (int b = 0; b < 4; ++b)
            if (i * 32 + b * 8 >= (i64)skip && i * 4 + b < end) v |= (u32)base[i * 4 + b] << (8 * b);
#endif
        if (i == 0) v &= ~0u << skip;
        return v;
    }
};
// bits sh .. sh + 63 of the three words
ZD_HD u64 join(u32 w0, u32 w1, u32 w2, u32 sh) {
    const u32 lo = (u32)((((u64)w1 << 32) | w0) >> sh), hi = (u32)((((u64)w2 << 32) | w1) >> sh);
    return ((u64)hi << 32) | lo;
}
// the top n bits of v, n <= 32
ZD_HD u32 top_bits(u64 v, u32 n) { return (u32)((v >> 1) >> (63u - n)); }

// ---- Huffman literals ----
// The weights of a tree description (RFC 8878 4.2.1) -> ws.w, their number -> nw; returns bytes used
// or < 0.  One thread.
template <class WS>
ZD_HD int read_huf_weights(const u8* src, u64 len, WS& ws, int& nw) {
    const u32 hb = src[0];
    nw = 0;
    if (hb < 128) {  // FSE-compressed weights, two interleaved states
        if (1 + hb > len) return kErrTruncated;
        int nsym = 0, log = 0;
        const int r = read_ncount(src + 1, hb, 6, 255, ws.norm[0], nsym, log);
        if (r < 0) return r;
        if (build_fse(ws.norm[0], nsym, log, ws.weights, ws.next) != kOk) return kErrFormat;
        const u8* p = src + 1 + r;
        const u64 bytes = hb - (u64)r;
        if (!bytes || !p[bytes - 1]) return kErrFormat;
        Words b;
        b.open(p, bytes);
        i64 pos = (i64)bytes * 8 - 8 + highbit(p[bytes - 1]);
        u64 v = 0;
        auto refill = [&]() {
            const i64 a = pos + (i64)b.skip - 64;
            v = join(b.word(a >> 5), b.word((a >> 5) + 1), b.word((a >> 5) + 2), (u32)a & 31u);
        };
        auto read = [&](u32 n) -> u32 {
            const u32 x = top_bits(v, n);
            v <<= n;
            pos -= n;
            return x;
        };
        refill();
        u32 s1 = read((u32)log), s2 = read((u32)log);
        for (u32 round = 1;; ++round) {  // at most 12 bits a round, 64 in the window
            if ((round & 3u) == 0) refill();
            if (nw >= 255) return kErrFormat;
            const FseEntry e1 = ws.weights[s1];
            ws.w[nw++] = e1.sym;
            s1 = e1.base + read(e1.nb);
            if (pos < 0) {
                ws.w[nw++] = ws.weights[s2].sym;
                break;
            }
            if (nw >= 255) return kErrFormat;
            const FseEntry e2 = ws.weights[s2];
            ws.w[nw++] = e2.sym;
            s2 = e2.base + read(e2.nb);
            if (pos < 0) {
                ws.w[nw++] = ws.weights[s1].sym;
                break;
            }
        }
        return (int)(1 + hb);
    }
    nw = (int)hb - 127;  // direct 4-bit weights
    const u64 nb = ((u64)nw + 1) / 2;
    if (1 + nb > len) return kErrTruncated;
    for (int i = 0; i < nw; ++i) ws.w[i] = (u8)((i & 1) ? (src[1 + i / 2] & 15) : (src[1 + i / 2] >> 4));
    return (int)(1 + nb);
}

// Tree description -> ws.huf; returns bytes used or < 0.
template <class WS, class Team>
ZD_HD int read_huf_tree(const u8* src, u64 len, WS& ws, int& huf_bits, const Team& team) {
    if (len < 1) return kErrTruncated;
    if (team.rank == 0) {
        int n = 0;
        ws.msg[0] = read_huf_weights(src, len, ws, n);
        ws.msg[1] = n;
    }
    team.sync();
    const int used = ws.msg[0], nw = ws.msg[1];
    if (used < 0) return used;
    if (nw > 255) return kErrFormat;  // 255 explicit weights at most: the implied one is the 256th
    // each weight's symbols are numbered in order, by one thread (0 and 13: none and too large)
    for (int k = team.rank; k < 14; k += team.size) {
        u32 c = 0;
        for (int i = 0; i < nw; ++i) {
            const int wi = ws.w[i];
            if (wi == k || (k == 13 && wi > kHufMaxBits + 1)) {
                ws.next[i] = (u16)c;
                ++c;
            }
        }
        ws.count[k] = c;
    }
    team.sync();
    // the last weight completes the sum to a power of two
    u32 sum = 0;
    for (int k = 1; k <= kHufMaxBits + 1; ++k) sum += ws.count[k] << (k - 1);
    if (ws.count[13] || !sum) return kErrFormat;
    const int maxb = highbit(sum) + 1;
    if (maxb > kHufMaxBits) return kErrFormat;
    const u32 rest = (1u << maxb) - sum;
    if (rest & (rest - 1)) return kErrFormat;
    const int last = highbit(rest) + 1;
    // symbols in order of increasing weight (the implied last one behind its equals), each of which
    // takes 2^(k-1) entries
    for (int i = team.rank; i <= nw; i += team.size) {
        const int k = i < nw ? ws.w[i] : last;
        if (!k) continue;
        u32 before = i < nw ? ws.next[i] : ws.count[k];
        for (int q = 1; q < k; ++q) before += ws.count[q] + (q == last ? 1u : 0u);
        ws.sorted[before] = (u8)i;
    }
    team.sync();
    for (u32 e = (u32)team.rank; e < 1u << maxb; e += (u32)team.size) {
        u32 first = 0, symbols = 0;
        int k = 1;
        for (; k <= maxb; ++k) {
            const u32 c = ws.count[k] + (k == last ? 1u : 0u);
            if (e < first + (c << (k - 1))) break;
            first += c << (k - 1);
            symbols += c;
        }
        ws.huf[e] = (u16)((ws.sorted[symbols + ((e - first) >> (k - 1))] << 8) | (maxb + 1 - k));
    }
    huf_bits = maxb;
    team.sync();
    return used;
}

// Decodes the n literals of a stream; one thread.
template <class WS>
ZD_HD int huf_stream(const u8* src, u64 len, u8* out, u64 n, const WS& ws, int mb) {
    BackBits bb;
    if (!bb.init(src, len)) return kErrFormat;
    for (u64 i = 0; i < n; ++i) {
        const u16 e = ws.huf[bb.peek(mb)];
        out[i] = (u8)(e >> 8);
        bb.pos -= (e & 0xff);
    }
    if (bb.pos != 0) return kErrFormat;
    return kOk;
}

// Literals of `streams` (1 or 4) Huffman streams: streams src[k], of len[k] bytes and n[k] literals, to
// out[k]; returns kOk or < 0, alike in every thread.  size / streams threads share a stream: each takes a
// piece of its bits, starts kHufWarm bits before it (codes fall in step with the true ones after a few
// symbols) and walks to its end, where the next thread's start has to be; a thread whose guess was wrong
// walks again from the true start.  With the counts each knows where its literals go and walks once more.
constexpr int kHufWarm = 192;
template <class WS, class Team>
ZD_HD int huf_streams_team(const u8* const* src, const u64* len, u8* const* out, const u64* n, int streams, WS& ws, int mb,
                           const Team& team) {
    const int L = team.size / streams, g = team.rank / L, j = team.rank % L;
    const u8* p = src[0];
    u64 bytes = len[0], want = n[0];
    u8* to = out[0];
    for (int q = 1; q < streams; ++q)
        if (g == q) {
            p = src[q];
            bytes = len[q];
            want = n[q];
            to = out[q];
        }
    BackBits bb;
    const bool ok = bb.init(p, bytes);
    const i64 total = ok ? bb.total : 0, piece = (total + L - 1) / L;
    const i64 top = total - j * piece > 0 ? total - j * piece : 0, floor = top - piece > 0 ? top - piece : 0;
    Words b;
    b.open(p, bytes);
    auto window = [&](i64 pos) -> u64 {
        const i64 a = pos + (i64)b.skip - 64;
        return join(b.word(a >> 5), b.word((a >> 5) + 1), b.word((a >> 5) + 2), (u32)a & 31u);
    };
    auto walk = [&](i64 pos, i64 down_to, u32& count) -> i64 {
        u32 c = 0;
        while (pos > down_to) {
            u64 v = window(pos);
            for (int u = 0; u < 5; ++u) {  // of at most 11 bits each
                if (pos <= down_to) break;
                const u32 bits = ws.huf[top_bits(v, (u32)mb)] & 0xffu;
                v <<= bits;
                pos -= bits;
                ++c;
            }
        }
        count += c;
        return pos;
    };
    u32 count = 0;
    i64 start = total;
    if (j > 0) start = walk(top + kHufWarm < total ? top + kHufWarm : total, top, count);
    bool walk_it = true;
    i64 stop = 0;
    for (;;) {  // at most L times: the first thread that was wrong is right afterwards
        if (walk_it) {
            count = 0;
            stop = walk(start, floor, count);
        }
        ws.end[team.rank] = stop;
        ws.num[team.rank] = count;
        team.sync();
        const i64 before = j ? ws.end[team.rank - 1] : total;
        walk_it = before != start;
        start = before;
        if (team.min(walk_it ? -1 : 0) == 0) break;
        team.sync();
    }
    u64 at = 0, all = 0;
    for (int q = 0; q < L; ++q) {
        const u32 c = ws.num[g * L + q];
        if (q < j) at += c;
        all += c;
    }
    const bool good = ok && ws.end[g * L + L - 1] == 0 && all == want;
    if (team.min(good ? 0 : kErrFormat) < 0) {
        team.sync();
        return kErrFormat;
    }
    i64 pos = start;
    u8* o = to + at;
    u32 acc = 0, held = 0, left = count;
    while (left) {
        u64 v = window(pos);
        for (int u = 0; u < 5; ++u) {
            if (!left) break;
            const u32 e = ws.huf[top_bits(v, (u32)mb)];
            v <<= e & 0xffu;
            pos -= e & 0xffu;
            --left;
            const u32 lane4 = (u32)((u64)o & 3u);
            acc |= (e >> 8) << (8u * lane4);
            ++held;
            ++o;
            if (lane4 == 3u || !left) {
#ifdef __CUDA_ARCH__
                if (held == 4) *reinterpret_cast<u32*>(o - 4) = acc;
                else
#endif
                    for (u32 q = 0; q < held; ++q) *(o - held + q) = (u8)(acc >> (8u * (lane4 + 1u - held + q)));
                acc = 0;
                held = 0;
            }
        }
    }
    team.sync();
    return kOk;
}

// Asks for src[0, n) ahead: on its way from memory into the L2 cache (near: the L1).
template <class Team>
ZD_HD void prefetch(const u8* src, u64 n, bool near, const Team& team) {
#ifdef __CUDA_ARCH__
    for (u64 i = 128u * team.rank; i < n; i += 128u * team.size) {
        if (near) asm volatile("prefetch.global.L1 [%0];" ::"l"(src + i));
        else asm volatile("prefetch.global.L2 [%0];" ::"l"(src + i));
    }
#endif
}

// dst[i] = src[i], eight in flight per thread; src does not reach into what is written.
template <class Team>
ZD_HD void copy_bytes(u8* dst, const u8* src, u64 n, const Team& team) {
    for (u64 i0 = team.rank; i0 < n; i0 += 8u * team.size) {
        u8 v[8];
#pragma unroll
        for (u32 k = 0; k < 8; ++k) v[k] = src[i0 + k * team.size < n ? i0 + k * team.size : n - 1];
#pragma unroll
        for (u32 k = 0; k < 8; ++k)
            if (i0 + k * team.size < n) dst[i0 + k * team.size] = v[k];
    }
}

// Literals section; returns bytes used or < 0.  lit: the nlit literals, for every thread.
template <class WS, class Team>
ZD_HD int read_literals(const u8* src, u64 len, WS& ws, int& huf_bits, const u8*& lit, u64& nlit, const Team& team) {
    team.sync();  // every thread is done with the previous block's literals
    lit = &ws.lit[0];
    if (len < 1) return kErrTruncated;
    const int type = src[0] & 3, fmt = (src[0] >> 2) & 3;
    if (type < 2) {
        u64 h, n;
        if (fmt == 0 || fmt == 2) {
            h = 1;
            n = src[0] >> 3;
        } else if (fmt == 1) {
            if (len < 2) return kErrTruncated;
            h = 2;
            n = (src[0] >> 4) | ((u32)src[1] << 4);
        } else {
            if (len < 3) return kErrTruncated;
            h = 3;
            n = (src[0] >> 4) | ((u32)src[1] << 4) | ((u32)src[2] << 12);
        }
        if (n > kMaxBlock) return kErrFormat;
        if (type == 0) {
            if (h + n > len) return kErrTruncated;
            lit = src + h;
            nlit = n;
            return (int)(h + n);
        }
        if (h + 1 > len) return kErrTruncated;
        for (u64 i = team.rank; i < n; i += team.size) ws.lit[i] = src[h];
        team.sync();
        nlit = n;
        return (int)(h + 1);
    }
    u64 h, regen, comp;
    int streams = fmt == 0 ? 1 : 4;
    if (fmt < 2) {
        if (len < 3) return kErrTruncated;
        const u32 v = rd24(src);
        h = 3;
        regen = (v >> 4) & 0x3ff;
        comp = (v >> 14) & 0x3ff;
    } else if (fmt == 2) {
        if (len < 4) return kErrTruncated;
        const u32 v = rd32(src);
        h = 4;
        regen = (v >> 4) & 0x3fff;
        comp = (v >> 18) & 0x3fff;
    } else {
        if (len < 5) return kErrTruncated;
        const u64 v = (u64)rd32(src) | ((u64)src[4] << 32);
        h = 5;
        regen = (v >> 4) & 0x3ffff;
        comp = (v >> 22) & 0x3ffff;
    }
    if (regen > kMaxBlock || h + comp > len) return kErrFormat;
    const u8* p = src + h;
    u64 rem = comp;
    if (type == 2) {
        const int r = read_huf_tree(p, rem, ws, huf_bits, team);
        if (r < 0) return r;
        p += r;
        rem -= (u64)r;
    } else if (!huf_bits) {
        return kErrFormat;  // repeated tree without a previous one
    }
    const u8* part[4] = {p, p, p, p};
    u64 size[4] = {rem, 0, 0, 0}, count[4] = {regen, 0, 0, 0};
    u8* to[4] = {&ws.lit[0], nullptr, nullptr, nullptr};
    if (streams == 4) {
        if (rem < 6) return kErrTruncated;
        const u64 s1 = rd16(p), s2 = rd16(p + 2), s3 = rd16(p + 4);
        if (6 + s1 + s2 + s3 > rem) return kErrTruncated;
        const u64 seg = (regen + 3) / 4;
        if (3 * seg > regen) return kErrFormat;
        size[0] = s1;
        size[1] = s2;
        size[2] = s3;
        size[3] = rem - 6 - s1 - s2 - s3;
        part[0] = p + 6;
        for (int k = 0; k < 4; ++k) {
            if (k) part[k] = part[k - 1] + size[k - 1];
            to[k] = &ws.lit[0] + (u64)k * seg;
            count[k] = k < 3 ? seg : regen - 3 * seg;
        }
    }
    int worst = kOk;
    if (team.size == 1) {
        for (int k = 0; k < streams; ++k) {
            const int r = huf_stream(part[k], size[k], to[k], count[k], ws, huf_bits);
            if (r < worst) worst = r;
        }
    } else {
        worst = huf_streams_team(part, size, to, count, streams, ws, huf_bits, team);
    }
    if (worst < 0) return worst;
    nlit = regen;
    return (int)(h + comp);
}

// The three sequence tables by their modes; returns bytes used or < 0.
template <class WS, class Team>
ZD_HD int read_tables(int modes, const u8* src, u64 len, WS& ws, Logs& lg, const Team& team) {
    constexpr int kMaxLog[3] = {9, 8, 9}, kMaxSym[3] = {35, 31, 52};
    if (team.rank == 0) {  // the descriptions, one after another
        int used = 0;
        for (int t = 0; t < 3 && used >= 0; ++t) {
            const int mode = (modes >> (6 - 2 * t)) & 3, max_log = t == 1 ? kMaxLog[1] : kMaxLog[0],
                      max_sym = t == 0 ? kMaxSym[0] : t == 1 ? kMaxSym[1] : kMaxSym[2];
            int nsym = 0, log = 0, r = 0;
            if (mode == 0) {
                if (t == 0) default_ll(ws.norm[0]);
                else if (t == 1) default_of(ws.norm[1]);
                else default_ml(ws.norm[2]);
                nsym = max_sym == 31 ? 29 : max_sym + 1;
                log = t == 1 ? 5 : 6;
            } else if (mode == 1) {  // one state, of one symbol
                if ((u64)used >= len) r = kErrTruncated;
                else if (src[used] > max_sym) r = kErrFormat;
                else {
                    nsym = src[used] + 1;
                    r = 1;
                }
            } else if (mode == 2) {
                r = read_ncount(src + used, len - (u64)used, max_log, max_sym, ws.norm[t], nsym, log);
            } else {
                log = lg.seq[t];
                if (log < 0) r = kErrFormat;
            }
            ws.built[t] = mode;
            ws.nsym[t] = nsym;
            ws.log[t] = log;
            used = r < 0 ? r : used + r;
        }
        ws.msg[2] = used;
        ws.msg[3] = kOk;
    }
    team.sync();
    const int used = ws.msg[2];
    if (used < 0) return used;
    // the states' symbols (RFC 8878 4.1.1), a thread per table
    for (int t = 0; t < 3; ++t) {
        if (team.rank != (team.size < 96 ? t % team.size : 32 * t)) continue;
        u8* sym = ws.state_sym[t];
        const short* norm = ws.norm[t];
        if (ws.built[t] == 1) sym[0] = (u8)(ws.nsym[t] - 1);
        if (ws.built[t] != 0 && ws.built[t] != 2) continue;
        const int size = 1 << ws.log[t], step = (size >> 1) + (size >> 3) + 3, mask = size - 1;
        int high = size - 1, p = 0;
        for (int s = 0; s < ws.nsym[t]; ++s)
            if (norm[s] == -1) sym[high--] = (u8)s;
        for (int s = 0; s < ws.nsym[t]; ++s) {
            const int c = norm[s];
            for (int i = 0; i < c; ++i) {
                sym[p] = (u8)s;
                do {
                    p = (p + step) & mask;
                } while (p > high);
            }
        }
        if (p != 0) ws.msg[3] = kErrFormat;
    }
    team.sync();
    if (ws.msg[3] < 0) return ws.msg[3];
    // the states of one symbol, in order, by one thread
    const int n0 = ws.built[0] == 3 ? 0 : ws.nsym[0], n1 = ws.built[1] == 3 ? 0 : ws.nsym[1],
              n2 = ws.built[2] == 3 ? 0 : ws.nsym[2];
    for (int q = team.rank; q < n0 + n1 + n2; q += team.size) {
        const int t = q < n0 ? 0 : q < n0 + n1 ? 1 : 2, s = t == 0 ? q : t == 1 ? q - n0 : q - n0 - n1;
        const int log = ws.log[t], size = 1 << log;
        u32 value = 0;
        int bits = s;
        if (t == 0) ll_code(s, value, bits);
        else if (t == 2) ml_code(s, value, bits);
        else value = 1u << s;
        const u32 extra = (u32)bits << 24;
        if (ws.built[t] == 1) {
            if (s == ws.nsym[t] - 1) {
                ws.seq_value[t][0] = value;
                ws.seq_next[t][0] = extra;
            }
            continue;
        }
        u32 ns = ws.norm[t][s] == -1 ? 1u : (u32)ws.norm[t][s];
        for (int i = 0; i < size; ++i) {
            if (ws.state_sym[t][i] != s) continue;
            const int nb = log - highbit(ns);
            ws.seq_value[t][i] = value;
            ws.seq_next[t][i] = ((ns << nb) - (u32)size) | ((u32)nb << 16) | extra;
            ++ns;
        }
    }
    for (int t = 0; t < 3; ++t) lg.seq[t] = ws.log[t];
    team.sync();
    return used;
}

// A sequence moves the last three offsets: each becomes one of them plus a number, or a number (RepMap:
// which << 32 | number; kRepConst: none of them).
constexpr u64 kRepConst = 3ull << 32;

// The first step of reading the n <= kBatch sequences next in the stream b, of whose bits `pos` are left:
// the states' chain, the only serial one.  Thread 0 walks it in staged bits and notes where each sequence
// starts.
ZD_HD int batch_base(const Words& b, int pos) { return ((pos + (int)b.skip + 31) >> 5) - kBatchWords; }
template <class WS, class Team>
ZD_HD void walk_states(const Words& b, int pos, int n, bool last, WS& ws, const Team& team) {
    const int base = batch_base(b, pos);
    u32 w[(kBatchWords + 2 + Team::size - 1) / Team::size];
#pragma unroll
    for (int i = 0; i < (kBatchWords + 2 + Team::size - 1) / Team::size; ++i) w[i] = b.word(base + team.rank + i * Team::size);
#pragma unroll
    for (int i = 0; i < (kBatchWords + 2 + Team::size - 1) / Team::size; ++i)
        if (team.rank + i * Team::size < kBatchWords + 2) ws.q_words[team.rank + i * Team::size] = w[i];
    team.sync();
    const int shift = (int)b.skip - 32 * base;  // staged bits are counted from q_words' first
    if (team.rank == 0) {
        u32 at = (u32)(pos + shift), s0 = ws.state[0], s1 = ws.state[1], s2 = ws.state[2];
        for (int c = 0; c < n; ++c) {
            const u32 e0 = ws.seq_next[0][s0], e1 = ws.seq_next[1][s1], e2 = ws.seq_next[2][s2];
            const u32 sum = e0 + e1 + e2;  // (the baselines are below 512: no carry)
            ws.q_at[c] = (u64)at | ((u64)(s0 | (s1 << 9) | (s2 << 18)) << 32);
            at -= sum >> 24;
            if (c + 1 == n && last) break;
            // state updates: literal length, match length, offset; 27 bits at most
            const u32 a = at - 32u;
            u32 x = (u32)((((u64)ws.q_words[(a >> 5) + 1] << 32) | ws.q_words[a >> 5]) >> (a & 31u));
            const u32 b0 = (e0 >> 16) & 0xffu, b1 = (e1 >> 16) & 0xffu, b2 = (e2 >> 16) & 0xffu;
            s0 = (e0 & 0xffffu) + ((x >> 1) >> (31u - b0));
            x <<= b0;
            s2 = (e2 & 0xffffu) + ((x >> 1) >> (31u - b2));
            x <<= b2;
            s1 = (e1 & 0xffffu) + ((x >> 1) >> (31u - b1));
            at -= (sum >> 16) & 0xffu;
        }
        ws.q_pos = at;
        ws.state[0] = s0;
        ws.state[1] = s1;
        ws.state[2] = s2;
    }
}

// The second step: the lengths and offsets are read by a thread each, and the repeated offsets and
// positions come by a scan; returns kOk or < 0.  Everything that the first step left is visible.
template <class WS, class Team>
ZD_HD int read_batch(const Words& b, int& pos, int n, u64 o, u64 cap, u64 literals_left, WS& ws, const Team& team) {
    pos = (int)ws.q_pos - (int)b.skip + 32 * batch_base(b, pos);
    if (team.rank == 0) ws.msg[0] = kOk;
    for (int c = team.rank; c < n; c += team.size) {
        const u32 st = (u32)(ws.q_at[c] >> 32), sl = st & 511u, so = (st >> 9) & 511u, sm = st >> 18;
        const u32 a = (u32)ws.q_at[c] - 64u, no = ws.seq_next[1][so] >> 24, nm = ws.seq_next[2][sm] >> 24, nl = ws.seq_next[0][sl] >> 24;
        const u64 v = join(ws.q_words[a >> 5], ws.q_words[(a >> 5) + 1], ws.q_words[(a >> 5) + 2], a & 31u);
        const u32 ofv = ws.seq_value[1][so] + top_bits(v, no), ml = ws.seq_value[2][sm] + top_bits(v << no, nm);
        const u32 ll = ws.seq_value[0][sl] + top_bits(v << (no + nm), nl);
        ws.q_ll[c] = ll;
        ws.q_len[0][c] = (u64)ll | ((u64)(ll + ml) << 32);
        const u32 idx = ofv > 3 ? 0u : ofv + (ll == 0 ? 1u : 0u);
        u64* const m = ws.q_rep[0][c];
        m[0] = idx == 0 ? kRepConst | (ofv - 3u) : idx == 4 ? (u64)0xffffffffu : (u64)(idx - 1u) << 32;
        m[1] = (u64)(idx == 1 ? 1u : 0u) << 32;
        m[2] = (u64)(idx == 1 || idx == 2 ? 2u : 1u) << 32;
    }
    // both by a scan of the batch, from buffer to buffer
    int at = 0;
    for (int d = 1; d < n; d <<= 1, at ^= 1) {
        team.sync();
        for (int c = team.rank; c < n; c += team.size) {
            const u64* const m = ws.q_rep[at][c];
            u64* const to = ws.q_rep[at ^ 1][c];
            for (int j = 0; j < 3; ++j) {
                const u64 x = m[j];
                const u64 y = ws.q_rep[at][c < d ? c : c - d][x >= kRepConst ? 0 : (int)(x >> 32)];
                to[j] = c < d || x >= kRepConst ? x : (y & ~0xffffffffull) | (u32)((u32)y + (u32)x);
            }
            ws.q_len[at ^ 1][c] = ws.q_len[at][c] + (c < d ? 0 : ws.q_len[at][c - d]);
        }
    }
    team.sync();
    auto offset = [&ws, at](int j, int c) -> u32 {  // the j-th last offset after the batch's sequence c
        const u64 x = ws.q_rep[at][c][j];
        return x >= kRepConst ? (u32)x : ws.rep[x >> 32] + (u32)x;
    };
    for (int c = team.rank; c < n; c += team.size) {
        ws.q_off[c] = offset(0, c);
        ws.q_start[c + 1] = (u32)(ws.q_len[at][c] >> 32);
        ws.q_lit[c + 1] = (u32)ws.q_len[at][c];
    }
    if (team.rank == 0) ws.q_start[0] = ws.q_lit[0] = 0;
    team.sync();
    if (team.rank == 0) {  // (read again in the next batch only)
        const u32 r0 = offset(0, n - 1), r1 = offset(1, n - 1), r2 = offset(2, n - 1);
        ws.rep[0] = r0;
        ws.rep[1] = r1;
        ws.rep[2] = r2;
    }
    if (ws.q_lit[n] > literals_left) return kErrFormat;
    if (ws.q_start[n] > cap - o) return kErrDstSize;  // (o <= cap)
    for (int c = team.rank; c < n; c += team.size)
        if (ws.q_off[c] == 0 || ws.q_off[c] > o + ws.q_start[c] + ws.q_ll[c]) ws.msg[0] = kErrFormat;
    team.sync();
    return ws.msg[0];
}

// The output of one sequence of any length.
template <class Team>
ZD_HD void run_long(u8* dst, const u8* lit, u32 ll, u32 off, u32 total, const Team& team) {
    copy_bytes(dst, lit, ll, team);
    team.sync();
    u8* const to = dst + ll;
    // byte i of a match repeats byte i mod off of the off bytes before it
    if (off >= total - ll) copy_bytes(to, to - off, total - ll, team);
    else
        for (u32 i = (u32)team.rank; i < total - ll; i += (u32)team.size) to[i] = *(to - off + i % off);
}

// The output of a chunk, the batch's sequences [first, last), at dst (of whose bytes those before it are
// visible; lit: the batch's first literal).  A byte is a
// literal, or repeats one before its sequence's match, which is before the chunk or in it.  Each thread
// takes eight bytes on an 8-byte boundary of the output and fetches those from outside the chunk; the
// others are followed, all at once, from byte to byte of the chunk until one of those.  (Copying sequence
// by sequence waits for a round trip through the L2 cache each time.)
template <class WS, class Team>
ZD_HD void run_chunk(WS& ws, int first, int last, u8* dst, const u8* lit, const Team& team) {
    const u32 begin = ws.q_start[first], total = ws.q_start[last] - begin;
    if (total > kChunkBytes) {
        run_long(dst, lit + ws.q_lit[first], ws.q_ll[first], ws.q_off[first], total, team);
        return;
    }
    const u32 lead = (u32)((u64)dst & 7u), groups = (lead + total + 7u) / 8u;
    u8* const value = reinterpret_cast<u8*>(ws.q_value);
    u16* const from = ws.q_from;
    bool inside = false;  // some byte of mine repeats one of the chunk
    for (u32 g = (u32)team.rank; g < groups; g += (u32)team.size) {
        const u32 lo = 8u * g > lead ? 8u * g - lead : 0u, hi = 8u * g + 8u - lead < total ? 8u * g + 8u - lead : total;
        int s = first;
        for (int d = 32; d; d >>= 1)
            if (s + d < last && ws.q_start[s + d] <= begin + lo) s += d;
        const u8* p8[8];
        u16 f8[8];
#pragma unroll
        for (u32 j = 0; j < 8; ++j) {
            const u32 x = 8u * g + j < lead ? lo : 8u * g + j - lead, p = x < hi ? x : hi - 1u;
            s += s + 1 < last && ws.q_start[s + 1] <= begin + p ? 1 : 0;  // (a sequence has 3 bytes at least)
            const u32 start = ws.q_start[s] - begin, r = p - start, ll = ws.q_ll[s], off = ws.q_off[s];
            // byte i of a match repeats byte i mod off of the off bytes before the match
            u32 i = r - ll;
            if (r >= ll && i >= off) i %= off;
            const i64 at = (i64)(start + ll + i) - (i64)off;
            const bool far = r < ll || at < 0;
            p8[j] = r < ll ? lit + ws.q_lit[s] + r : dst + (at < 0 ? at : 0);
            f8[j] = (u16)(lead + (far ? p : (u32)at));
            inside |= !far;
        }
        u64 v = 0, f0 = 0, f1 = 0;
#pragma unroll
        for (u32 j = 0; j < 8; ++j) {
            v |= (u64)*p8[j] << (8u * j);
            if (j < 4) f0 |= (u64)f8[j] << (16u * j);
            else f1 |= (u64)f8[j] << (16u * (j - 4u));
        }
        ws.q_value[g] = v;
        memcpy(__builtin_assume_aligned(from + 8u * g, 8), &f0, 8);
        memcpy(__builtin_assume_aligned(from + 8u * g + 4u, 8), &f1, 8);
    }
    team.sync();
    // a byte's source may meanwhile have been replaced by a later one on the same way: as good
    while (inside) {
        inside = false;
        for (u32 g = (u32)team.rank; g < groups; g += (u32)team.size)
            for (u32 j = 0; j < 8; ++j) {
                const u16 a = from[8u * g + j], b = from[a];
                if (a != b) {
                    from[8u * g + j] = b;
                    inside = true;
                }
            }
    }
    for (u32 g = (u32)team.rank; g < groups; g += (u32)team.size) {
        const u32 lo = 8u * g > lead ? 8u * g - lead : 0u, hi = 8u * g + 8u - lead < total ? 8u * g + 8u - lead : total;
        u64 v = 0;
#pragma unroll
        for (u32 j = 0; j < 8; ++j) v |= (u64)value[from[8u * g + j]] << (8u * j);
#ifdef __CUDA_ARCH__
        if (hi - lo == 8u) {
            *reinterpret_cast<u64*>(dst + lo) = v;
            continue;
        }
#endif
        const u32 skip = 8u * g + 8u > lead && 8u * g < lead ? lead - 8u * g : 0u;
        for (u32 j = 0; j < hi - lo; ++j) dst[lo + j] = (u8)(v >> (8u * (skip + j)));
    }
}

// One compressed block into dst[op ...]; returns bytes written or < 0.
template <class WS, class Team>
ZD_HD i64 decode_block(const u8* src, u64 len, u8* dst, u64 op, u64 cap, WS& ws, Logs& lg,
                       const Team& team) {
    u64 nlit = 0;
    const u8* lit = nullptr;
    const int lr = read_literals(src, len, ws, lg.huf_bits, lit, nlit, team);
    if (lr < 0) return lr;
    const u8* p = src + lr;
    u64 rem = len - (u64)lr;
    if (rem < 1) return kErrTruncated;
    u64 nseq;
    if (p[0] == 0) {
        nseq = 0;
        p += 1;
        rem -= 1;
    } else if (p[0] < 128) {
        nseq = p[0];
        p += 1;
        rem -= 1;
    } else if (p[0] < 255) {
        if (rem < 2) return kErrTruncated;
        nseq = ((u64)(p[0] - 128) << 8) + p[1];
        p += 2;
        rem -= 2;
    } else {
        if (rem < 3) return kErrTruncated;
        nseq = (u64)p[1] + ((u64)p[2] << 8) + 0x7f00;
        p += 3;
        rem -= 3;
    }
    u64 o = op;
    if (nseq == 0) {
        if (o + nlit > cap) return kErrDstSize;
        copy_bytes(dst + o, lit, nlit, team);
        return (i64)nlit;
    }
    if (rem < 1) return kErrTruncated;
    const int modes = p[0];
    p += 1;
    rem -= 1;
    const int r = read_tables(modes, p, rem, ws, lg, team);
    if (r < 0) return r;
    p += r;
    rem -= (u64)r;
    if (!rem || !p[rem - 1]) return kErrFormat;
    prefetch(p, rem, true, team);
    Words b;
    b.open(p, rem);
    int pos = (int)rem * 8 - 8 + highbit(p[rem - 1]);  // bits left (a block is below 2^17 bytes)
    if (team.rank == 0) {
        const i64 a = (i64)pos + (i64)b.skip - 64;
        u64 v = join(b.word(a >> 5), b.word((a >> 5) + 1), b.word((a >> 5) + 2), (u32)a & 31u);
        for (int t = 0; t < 3; ++t) {
            ws.state[t] = top_bits(v, (u32)ws.log[t]);
            v <<= ws.log[t];
        }
    }
    pos -= ws.log[0] + ws.log[1] + ws.log[2];
    u64 li = 0;
    auto batch = [&](u64 k) { return nseq - k < (u64)kBatch ? (int)(nseq - k) : kBatch; };
    // the batch's sequences from the first on, as many as make a chunk at a time
    auto run = [&](int n, const auto& some) {
        for (int first = 0; first < n;) {
            int next = first;
            for (int d = 32; d; d >>= 1)
                if (next + d <= n && ws.q_start[next + d] - ws.q_start[first] <= kChunkBytes) next += d;
            next += next < n && ws.q_start[next + 1] - ws.q_start[first] <= kChunkBytes ? 1 : 0;  // (the 64th)
            if (next == first) ++next;
            if (first) some.sync();  // the chunk before is visible, and every thread has done with it
            run_chunk(ws, first, next, dst + o + ws.q_start[first], lit + li, some);
            first = next;
        }
    };
    team.sync();
    walk_states(b, pos, batch(0), (u64)batch(0) == nseq, ws, team);
    for (u64 k = 0; k < nseq; k += kBatch) {
        team.sync();
        const int n = batch(k);
        const int e = read_batch(b, pos, n, o, cap, nlit - li, ws, team);
        if (e < 0) return e;
        const u64 after = k + (u64)n;
#ifdef __CUDA_ARCH__
        // one warp walks the next batch's states while the others write this one's output
        if (team.rank < 32) {
            if (after < nseq) walk_states(b, pos, batch(after), after + (u64)batch(after) == nseq, ws, HeadTeam{team.rank});
        } else {
            run(n, TailTeam{team.rank - 32});
        }
#else
        run(n, team);
        team.sync();
        if (after < nseq) walk_states(b, pos, batch(after), after + (u64)batch(after) == nseq, ws, team);
#endif
        team.sync();
        li += ws.q_lit[n];
        o += ws.q_start[n];
    }
    if (pos != 0) return kErrFormat;
    if (o + (nlit - li) > cap) return kErrDstSize;
    copy_bytes(dst + o, lit + li, nlit - li, team);
    o += nlit - li;
    return (i64)(o - op);
}

// One frame: src[0..len) -> dst[0..cap); returns the content size or < 0.
template <class WS, class Team>
ZD_HD i64 decode_frame(const u8* src, u64 len, u8* dst, u64 cap, WS& ws, const Team& team) {
    if (len < 6 || rd32(src) != 0xFD2FB528u) return kErrFormat;
    const u32 fhd = src[4];
    const int fcs_flag = fhd >> 6, single = (fhd >> 5) & 1, checksum = (fhd >> 2) & 1, did = fhd & 3;
    if (fhd & 8) return kErrFormat;  // reserved bit
    u64 p = 5;
    if (!single) p += 1;  // window descriptor
    const int did_bytes = did == 0 ? 0 : did == 1 ? 1 : did == 2 ? 2 : 4;
    if (did_bytes) return kErrFormat;  // dictionaries are not used by the container frames
    const int fcs_bytes = fcs_flag == 0 ? (single ? 1 : 0) : fcs_flag == 1 ? 2 : fcs_flag == 2 ? 4 : 8;
    if (p + fcs_bytes > len) return kErrTruncated;
    u64 fcs = ~0ull;
    if (fcs_bytes == 1) fcs = src[p];
    else if (fcs_bytes == 2) fcs = rd16(src + p) + 256;
    else if (fcs_bytes == 4) fcs = rd32(src + p);
    else if (fcs_bytes == 8) fcs = (u64)rd32(src + p) | ((u64)rd32(src + p + 4) << 32);
    p += fcs_bytes;
    prefetch(src, len, false, team);
    Logs lg;
    if (team.rank == 0) {
        ws.rep[0] = 1;
        ws.rep[1] = 4;
        ws.rep[2] = 8;
    }
    u64 o = 0;
    for (;;) {
        if (p + 3 > len) return kErrTruncated;
        const u32 bh = rd24(src + p);
        p += 3;
        const int last = bh & 1, type = (bh >> 1) & 3;
        const u64 bsize = bh >> 3;
        if (type == 3) return kErrFormat;
        if (type == 0) {
            if (p + bsize > len) return kErrTruncated;
            if (o + bsize > cap) return kErrDstSize;
            copy_bytes(dst + o, src + p, bsize, team);
            o += bsize;
            p += bsize;
        } else if (type == 1) {
            if (p + 1 > len) return kErrTruncated;
            if (o + bsize > cap) return kErrDstSize;
            for (u64 i = team.rank; i < bsize; i += team.size) dst[o + i] = src[p];
            o += bsize;
            p += 1;
        } else {
            if (bsize > kMaxBlock || p + bsize > len) return kErrTruncated;
            const i64 w = decode_block(src + p, bsize, dst, o, cap, ws, lg, team);
            if (w < 0) return w;
            o += (u64)w;
            p += bsize;
        }
        if (last) break;
    }
    if (checksum) p += 4;
    if (p > len) return kErrTruncated;
    if (fcs != ~0ull && fcs != o) return kErrFormat;
    return (i64)o;
}

}  // namespace zd
}  // namespace xnyz
