// Launchers of the sm_100a kernels (implemented in k_*.cu), called by the host pipeline.
// All pointers are device pointers unless named *_host; every launcher is asynchronous on
// `st`.  Plain C++ types only, so host .cpp files include this without CUDA headers.
#pragma once

#include <cstddef>
#include <cstdint>

typedef struct CUstream_st* cudaStream_t;

namespace xnyz {
namespace dev {

struct QuantParams {
    int quantizer;  // 0 cube, 1 truncated octahedron, 2 adaptive
    float div;      // float(double(2*l2)/sqrt(3|5))
    float s;        // l2 as float
    float rdiv;     // float(sqrt(3|5))
    float inv;      // 1 / div correctly rounded, or 0: divide (quantize_range_kernel checks the extents too)
    float rinv;     // 1 / rdiv correctly rounded, or 0: divide (a bound near the float range's ends)
    float step[3];  // adaptive: per-axis steps (decompression: from the container)
    const float* step_dev;  // adaptive compression: the steps in device memory (PointStats::step)
};

// Results of the bounding-box / quantization sweeps (one struct in device memory).
struct PointStats {
    unsigned long long minkey[3];  // per axis: (order key << 32) | first index of the minimum
    int max_cell[3];               // max lattice index per axis (>= 0: starts at 0 like the reference)
    int min_cell[3];               // min lattice index per axis (starts at INT_MAX)
    unsigned int nonfinite;        // inputs that are NaN or +-inf
    unsigned int mse_max_bits;     // max per-point squared error (float bits)
    double mse_sum;                // sum of per-point squared errors
    unsigned int err;              // device error bits
    float offset[3];               // shift offset (written by quantize_range)
    unsigned int maxkey[3];        // per axis: largest order key (bbox, for the adaptive steps)
    float step[3];                 // adaptive quantizer steps (launch_adaptive_steps)
};

// Key layout of block mode.  Normal cells: key = id << 21 | quad << 18 | sfc18.  Cells with
// z = -1 (the truncated-octahedron edge case) carry `defect_flag` and the id minus
// `defect_base` so that they sort after all other cells in the reference's id order.
struct BlockKeyParams {
    unsigned long long nx, nxy;      // blocks per row, per layer (nx < 2^25)
    unsigned long long defect_flag;  // 0 if no z = -1 cells
    unsigned long long defect_base;  // ((2^64-1)/64/2) * nx * ny  (mod 2^64)
    int hilbert;
    unsigned int hstart;  // Hilbert state after levels 20..6 (all zero digits)
};

// Key layout of direct mode: key = sfc, or defect_flag | (sfc & (defect_flag - 1)) for z = -1
// cells whose high sfc bits equal `defect_high`.
struct DirectKeyParams {
    int bits;      // hilbert_bits = bit length of the max range (>= 1)
    int hilbert;
    unsigned long long defect_flag;
    unsigned long long defect_high;
};

// Unit (unique cell, or point for -normal) outputs of the segment kernels.
struct UnitOutputs {
    uint8_t* rep_sym;               // PFor symbol of repos / sfc delta per unit
    uint8_t* quad_sym;              // PFor symbol of the quad delta per unit (block mode)
    void* patches;                  // PFor patches in order: u32 in block mode (18-bit codes), u64 in direct mode
    unsigned long long* blk_id;     // block mode: id of each block
    uint32_t* blk_unit;             // block mode: first unit of each block
    uint32_t* unit_pos;             // -rle: sorted position of each unit's first point
    unsigned long long* hist_rep;   // [256]
    uint32_t* first_rep;            // [256]
    unsigned long long* hist_quad;  // [256]
    uint32_t* first_quad;           // [256]
    unsigned long long* counters;   // [0] units, [1] patches, [2] blocks, [3] sum of patches
    unsigned long long* rep_val;    // optional: repos / sfc delta value per unit (extended container)
};

// State of a chained scan: 16 bytes per tile, zeroed (device_common.cuh: chain_lookback).
using ScanStatus = void*;
constexpr size_t kScanStatusBytes = 16;

// Count-stream statistics (-rle).
constexpr int kCountDense = 4096;
struct CountStats {
    struct Bin {                // of counts below kCountDense
        unsigned long long n;
        uint32_t inv_first;     // ~(first unit with this count), 0 when none
        uint32_t unused;
    };
    Bin* bins;                  // [kCountDense]
    uint32_t* max_dense;        // largest such count
    uint32_t* over_val;         // counts >= kCountDense: value
    uint32_t* over_unit;        //   ... and unit index
    uint32_t* over_n;           // number of such counts
};

// Huffman code table for uint8 symbols, and for int counts (dense part + sorted sparse part).
struct ByteCodes {
    uint32_t bits[256];
    uint8_t len[256];
};

struct EncodeTotals {
    unsigned long long bits[8];  // total bits per stream (see Stream enum in pipeline.cpp)
};

// --- points ---------------------------------------------------------------------------
void launch_bbox(const float* xyz, uint64_t n, PointStats* stats, cudaStream_t st);
// AdaptiveQuantizer steps from the bounding box (after launch_bbox) into stats->step.
void launch_adaptive_steps(const float* xyz, float l2, PointStats* stats, cudaStream_t st);
// cells (optional, 3 n int32): each finite point's lattice cell, for launch_keys_cells.
void launch_quantize_range(const float* xyz, uint64_t n, QuantParams q, PointStats* stats, int with_error_stats,
                           cudaStream_t st, int32_t* cells = nullptr);
void launch_keys_direct(const float* xyz, uint64_t n, QuantParams q, const PointStats* stats, DirectKeyParams kp,
                        const uint8_t* hilbert_tab, unsigned long long* keys, uint32_t* payload, int passes,
                        uint32_t* hist, cudaStream_t st);
// Cell tables: block keys from int32 cells; per-axis min / max of cells (stats->min_cell /
// max_cell, initialised by the caller); dst[i] = src[idx[i]]; expansion + recover + unshift
// (status: ceil(n / 4096) tiles; *total receives the point count).
void launch_keys_cells(const int32_t* cells, uint64_t n, BlockKeyParams kp, const uint16_t* hilbert_fwd2,
                       unsigned long long* keys, uint32_t* payload, int passes, uint32_t* hist, cudaStream_t st);
void launch_cells_stats(const int32_t* cells, uint64_t n, PointStats* stats, cudaStream_t st);
void launch_gather_i32(const int32_t* src, const uint32_t* idx, uint64_t n, int32_t* dst, cudaStream_t st);
void launch_expand_cells(const int32_t* cells, const int32_t* counts, uint64_t n, QuantParams q, const float* off3,
                         ScanStatus status, uint32_t* tile_counter, float* out, uint64_t cap,
                         unsigned long long* total, uint32_t* err, cudaStream_t st);
void launch_quantize_cells(const float* xyz, uint64_t n, QuantParams q, const PointStats* stats, int32_t* cells,
                           cudaStream_t st);
void launch_recover_cells(const int32_t* cells, uint64_t n, QuantParams q, const float* offset3_dev, float* xyz,
                          cudaStream_t st);
void launch_hilbert(const unsigned long long* in, uint64_t n, const uint8_t* tab, int top, unsigned int state,
                    unsigned long long* out, cudaStream_t st);

// --- sort -----------------------------------------------------------------------------
// Keys per block of a pass: small arrays take small tiles, so that they still cover the 148 SMs
// (1M keys: 244 tiles of 4096, 120K: 59 of 2048).  At most 256 tiles up to 2^20 keys.
constexpr uint32_t sort_tile(uint64_t n) { return n <= 256u * 2048 ? 2048u : n <= 256u * 4096 ? 4096u : 8192u; }
constexpr uint64_t sort_tiles(uint64_t n) { return (n + sort_tile(n) - 1) / sort_tile(n); }
void launch_sort_histogram(const unsigned long long* keys, uint64_t n, int passes, uint32_t* hist, cudaStream_t st);
void launch_sort_offsets(uint32_t* hist, int passes, cudaStream_t st);  // in place: counts -> exclusive offsets
void launch_sort_pass(const unsigned long long* kin, unsigned long long* kout, const uint32_t* vin, uint32_t* vout,
                      uint64_t n, int shift, const uint32_t* offsets, unsigned long long* status, uint32_t epoch,
                      uint32_t* tile_counter, uint32_t* err, cudaStream_t st);
// All passes of up to kSortSmall keys in one launch; the output may be the input.
constexpr uint64_t kSortSmall = 8192;
void launch_sort_small(const unsigned long long* kin, unsigned long long* kout, const uint32_t* vin, uint32_t* vout,
                       uint64_t n, int passes, cudaStream_t st);

// --- compress segments + encoders -------------------------------------------------------
constexpr int kUnitTile = 4096, kUnitTileSmall = 1024;
constexpr uint64_t kUnitSmall = 1ull << 19;
inline uint64_t unit_tile(uint64_t n) { return n < kUnitSmall ? kUnitTileSmall : kUnitTile; }
void launch_units_block(const unsigned long long* keys, uint64_t n, int rle, BlockKeyParams kp, UnitOutputs out,
                        ScanStatus status, uint32_t* tile_counter, uint32_t* err, cudaStream_t st);
void launch_units_direct(const unsigned long long* keys, uint64_t n, int rle, DirectKeyParams kp, UnitOutputs out,
                         ScanStatus status, uint32_t* tile_counter, uint32_t* err, cudaStream_t st);
// unit_pos null: counts[] is the input (cell tables), else counts[] receives the run lengths.
void launch_count_stats(const uint32_t* unit_pos, uint64_t units, const unsigned long long* units_dev, uint64_t n,
                        int32_t* counts, CountStats cs, cudaStream_t st);
// Largest block-id delta and block-count delta, into max2[0] and max2[1].  counters[0] and [2] (device)
// hold the units and blocks; most_blocks bounds the latter.
void launch_block_max(const unsigned long long* blk_id, const uint32_t* blk_unit, uint64_t most_blocks,
                      const unsigned long long* counters, unsigned long long* max2, cudaStream_t st);
// Bit-packs the block-id and block-count deltas (widths 1..64).  Widths from 8 on: written to the
// ceil(nblocks width / 8) bytes at dst (any alignment), nothing else touched; narrower: OR-ed into
// the zeroed words at `words`.
struct BlockPackDst {
    uint8_t* dst;
    uint32_t* words;
    int width;
};
constexpr int kPackDirectWidth = 8;
void launch_block_pack(const unsigned long long* blk_id, const uint32_t* blk_unit, uint64_t nblocks, uint64_t units,
                       const BlockPackDst& blk, const BlockPackDst& cnt, cudaStream_t st);

// Lays pieces of any alignment out at dst + off in one launch: device memory, bytes of the argument
// itself, zeros, and one stream whose length only the device knows (ceil(*late_bits / 8), at most
// late_most): its length as 8 bytes and its data.  Pieces with `after` lie that much further on.
constexpr int kGatherPieces = 24;
constexpr size_t kGatherInline = 4096;
enum { kGatherCopy, kGatherInlineBytes, kGatherZero, kGatherLateLen, kGatherLate };
struct GatherPiece {
    const uint8_t* src;
    uint64_t off, len;
    uint32_t inline_off;
    uint8_t kind, after;
};
struct GatherArgs {
    GatherPiece piece[kGatherPieces];
    int count;
    const unsigned long long* late_bits;
    uint64_t late_most;
    uint8_t inline_bytes[kGatherInline];
};
void launch_gather(const GatherArgs& args, uint8_t* dst, cudaStream_t st);

constexpr int kEncTile = 4096;
// One entropy coder of launch_encode.  It writes at most cap_bits bits (the output buffer's size; words
// zeroed) and flags an overflow beyond; *total_bits receives the bits written.
enum { kEncodeGolombRice32, kEncodeGolombRice64, kEncodeHuffman, kEncodeFixedU8, kEncodeFixedI32, kEncodeCounts };
struct EncodeJob {
    int kind;
    // Golomb-Rice parameter; fixed-length codes: the length (1..24); counts: exp-Golomb parameter, or
    // -1 for Huffman
    int k;
    const void* in;  // n values: u32 / u64 (Golomb-Rice), u8 symbols, i32 counts; 16-byte aligned
    uint64_t n;
    const ByteCodes* codes;  // kEncodeHuffman
    // fixed-length codes and counts: code bits by symbol (at least 256 entries; counts: a dense table
    // [kCountDense], with lengths, and sorted sparse values)
    const uint32_t* bits;
    const uint8_t* len;
    const uint32_t *sparse_val, *sparse_bits;
    const uint8_t* sparse_len;
    uint32_t sparse_n;
    uint32_t blocks;  // set by launch_encode
    uint32_t* words;
    uint64_t cap_bits;
    ScanStatus status;
    uint32_t* tile_counter;
    unsigned long long* total_bits;
};
struct EncodeArgs {
    EncodeJob job[4];
    int count;
    uint32_t* err;
};
void launch_encode(EncodeArgs args, cudaStream_t st);

// Sets ranges of words in one launch.
struct FillRange {
    void* p;  // 4-byte aligned
    uint64_t words;
    uint32_t value;
};
struct FillArgs {
    FillRange range[24];
    int count;
};
void launch_fill(const FillArgs& args, cudaStream_t st);

// --- decompress -------------------------------------------------------------------------

// Parallel decoding of one unindexed prefix-code stream (Huffman, Golomb-Rice, exp-Golomb),
// implemented in k_stream_decode.cu.
enum CodeKind { kCodeHuffman = 0, kCodeGolombRice = 1, kCodeExpGolomb = 2 };
struct DecodeTable {
    // Huffman: primary table of 2^root_bits entries (1 <= root_bits <= 11): (len << 24) |
    // payload for codes of at most root_bits bits, 0 for a prefix that is no code,
    // (1u << 31) | node for longer codes; tree nodes hold two children each (leaf =
    // (1u << 31) | payload, internal = node index, missing = 0xffffffff).  The payload is
    // the symbol value when symvals is null, else an index into symvals.
    const uint32_t* root;
    const uint32_t* tree;
    const unsigned long long* symvals;
    int root_bits;
    int param;   // Golomb-Rice / exp-Golomb k
    int zigzag;  // exp-Golomb of a signed symbol type
};
constexpr int kDecodeMaxL = 64;       // longest entry offset tracked per subsequence
constexpr int kDecodeSubBits = 512;   // bits per subsequence (thread): Huffman, exp-Golomb
constexpr int kDecodeSubBitsGR = 1024;  // Golomb-Rice (longer subsequences amortise its entry tables)
constexpr int kDecodeBlockSubs = 128; // subsequences per thread block
// flag: [tiles]; agg: [tiles * kDecodeMaxL]; inc: [tiles * 2];
// tiles = ceil(ceil(bits / sub bits) / kDecodeBlockSubs) (kDecodeSubBits, the smaller, bounds
// the tiles of every kind).
// The stream starts `base_bits` (< 32) into `words`.  L = entry offsets tracked (the longest
// codeword; Golomb-Rice derives k + 2 from its parameter).
void launch_decode_stream(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits, DecodeTable t,
                          int L, uint64_t nsym, int out_width, void* out, uint32_t* flag,
                          unsigned long long* agg, unsigned long long* inc, uint32_t* tile_counter, uint32_t* err,
                          uint32_t* need_fallback, unsigned long long* total_codewords, cudaStream_t st);
// Self-synchronising decoder: needs no entry tables, for streams whose decoding falls in step
// from any bit offset.  *need_fallback (starts at 0) tells why the stream has to be decoded
// otherwise: 1 a bounded wait expired, 2 it did not fall in step, 4 a Golomb-Rice value of 2^32 or
// more with out_width 4.  status: 16 bytes per tile, zeroed, 16-byte aligned; *redone starts at 0.
// out: 16-byte aligned.  byte_symbols: every symbol value is below 256.
struct SyncGeometry {
    int S;           // bits per subsequence
    int G;           // subsequences a block decodes ahead of its own
    uint64_t tiles;  // blocks
};
SyncGeometry sync_geometry(int kind, uint64_t total_bits);
void launch_decode_sync(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits, DecodeTable t,
                        bool byte_symbols, uint64_t nsym, int out_width, void* out, void* status,
                        uint32_t* tile_counter, uint32_t* err, uint32_t* need_fallback, uint32_t* redone,
                        unsigned long long* total_codewords, cudaStream_t st);
// A Huffman stream whose codewords all have length len (== t.root_bits <= 11): every symbol
// from its own len bits (out_width 1: u8, 4: u32 values).
void launch_decode_fixed(const uint32_t* words, uint64_t base_bits, uint64_t total_bits, DecodeTable t, int len,
                         uint64_t nsym, int out_width, void* out, uint32_t* err, cudaStream_t st);
// One-thread decoder the host runs when a bounded wait of a parallel decoder expired.
void launch_decode_sequential(int kind, const uint32_t* words, uint64_t base_bits, uint64_t total_bits,
                              DecodeTable t, uint64_t nsym, int out_width, void* out,
                              unsigned long long* total_codewords, uint32_t* err, cudaStream_t st);
void launch_fill_u8(uint8_t* p, uint64_t n, uint8_t v, cudaStream_t st);
void launch_fill_u32(uint32_t* p, uint64_t n, uint32_t v, cudaStream_t st);

// Division of any 64-bit value by an invariant divisor d >= 1 through one high multiply
// (T. Granlund and P. Montgomery, "Division by invariant integers using multiplication",
// PLDI 1994, section 4, figure 4.1): with l = ceil(log2 d) and m = floor(2^64 (2^l - d) / d)
// + 1, x / d = (t + ((x - t) >> min(l, 1))) >> max(l - 1, 0) where t = mulhi(m, x).  For x below
// 2^44 (all block ids but those of z = -1 cells) the same theorem with N = 44 needs no correction:
// x / d = mulhi(x << 20, m44) >> l with m44 = ceil(2^(44 + l) / d).
struct U64Div {
    unsigned long long m, m44;
    unsigned int sh1, sh2, l44;
};
inline U64Div make_u64div(unsigned long long d) {
    unsigned int l = 0;
    while (l < 64 && (static_cast<unsigned __int128>(1) << l) < d) ++l;
    const unsigned __int128 num = (static_cast<unsigned __int128>(1) << 64) *
                                  ((static_cast<unsigned __int128>(1) << l) - d);
    U64Div r;
    r.m = static_cast<unsigned long long>(num / d + 1);
    r.sh1 = l < 1 ? l : 1;
    r.sh2 = l > 1 ? l - 1 : 0;
    r.m44 = static_cast<unsigned long long>(((static_cast<unsigned __int128>(1) << (44 + l)) + d - 1) / d);
    r.l44 = l < 63 ? l : 63;
    return r;
}

// LCP recovery (block mode) or SFC prefix sum (direct mode) fused with the PFor decode,
// -rle expansion, recover and unshift.
struct RecoverParams {
    QuantParams q;
    float off[3];
    int hilbert;
    unsigned int hstart_inv;  // inverse-Hilbert state after levels 20..6 of zero digits
    int rle;
    int direct;
    int bits;   // direct mode hilbert_bits
    int cells;  // write the units' int32 lattice cells instead of points (no expansion, no recover)
};
// Lattice corner of each block that has units, in order.
struct BlockCorners {
    uint32_t *x, *y, *z;
};
// What comes before a tile of kRecoverTile units: patches (zero symbols), block starts, outputs.
struct TilePrefix {
    uint32_t zeros, starts;
    unsigned long long outputs;
};
struct RecoverInputs {
    const TilePrefix* prefix;      // per tile and one past the last (launch_tile_prefix)
    const uint8_t* rep_sym;        // byte arrays: 8-byte aligned, readable 8 bytes past the end
    const void* rep_patch;         // Golomb-Rice decoded patches: u32 when patch32, else u64
    int patch32;
    uint64_t npatch;
    const uint8_t* quad_sym;
    const uint8_t* is_start;       // block mode: 1 where a non-empty block starts
    BlockCorners corners;
    uint64_t nblocks;
    const int32_t* counts;         // -rle: 16-byte aligned, readable 32 bytes past the end
    const unsigned long long* rep_val;  // extended container: repos / sfc delta per unit (replaces rep_sym + patches)
};
// Collects a container's header bytes (the fixed fields, every stream's lengths and meta, the trailing
// offset) into pinned host memory at `out`: HeaderPieces, then the bytes.  Stops at lengths that leave
// the container.
struct HeaderPieces {
    uint32_t count, unused;
    struct {
        uint64_t off;      // in the container
        uint32_t len, at;  // bytes collected, and where after the struct
    } piece[10];
};
constexpr size_t kHeaderBytes = 32768;
// First 8 bytes of an extended container ("XNYZBX01"): the reference container follows,
// except that the repos / SFC-delta stream is block-coded (k_blocks.cu).
constexpr uint64_t kExtendedMagic = 0x313058425a594e58ull;
void launch_header(const uint8_t* cont, uint64_t len, int rle, uint8_t* out, cudaStream_t st);

// Block streams of block mode in one pass: bit-unpack (widths <= 64), inclusive prefix sums of
// the block-id and block-count deltas, block-start marks (is_start zeroed by the caller) and corners.
// Sets *empty when a block has no units: then call again with `compact` (everything zeroed again).
// The words of each stream are read from the 16-byte boundary before its first to the one after the
// 12 bytes past its last.  status: [3][tiles], tiles = ceil(nblocks / kBlockStreamTile).
constexpr int kBlockStreamTile = 2048;
void launch_block_streams(const uint32_t* words_blk, uint64_t base_blk, int width_blk, const uint32_t* words_cnt,
                          uint64_t base_cnt, int width_cnt, uint64_t nblocks, uint64_t units, uint64_t nx, uint64_t ny,
                          bool compact, BlockCorners corners, uint8_t* is_start, ScanStatus status, uint32_t* tile_counter,
                          unsigned long long* count_total, uint32_t* empty, uint32_t* err, cudaStream_t st);
constexpr int kRecoverTile = 2048;
// Prefixes of the recover tiles, and the outputs' number; null inputs count nothing (rep_sym: no patches,
// is_start: direct mode, counts: -normal).  status: one word per kPrefixTiles tiles.
constexpr int kPrefixTiles = 4;
void launch_tile_prefix(const uint8_t* rep_sym, const uint8_t* is_start, const int32_t* counts, uint64_t units,
                        TilePrefix* out, ScanStatus status, uint32_t* tile_counter, unsigned long long* count_total,
                        uint32_t* err, cudaStream_t st);
// status: [tiles], tiles = ceil(units / kRecoverTile); hilbert_inv2: two levels of the inverse
// machine per entry ([32][64]: x | y << 2 | z << 4 | next state << 6)
void launch_recover_units(const RecoverInputs& in, uint64_t units, uint64_t nout, RecoverParams rp,
                          const uint8_t* hilbert_inv_tab, const uint16_t* hilbert_inv2, ScanStatus status,
                          uint32_t* tile_counter, float* out, uint32_t* err, cudaStream_t st);

// --- block-parameter coding (extended container) and its predictor ------------------------
constexpr int kParamBlock = 1024;     // values per block
constexpr int kParamFeatures = 34;    // features per block (row stride of the feature array)
constexpr int kParamInputs = 34;
constexpr int kParamOutputsK = 32;    // Golomb-Rice k in 0..31
constexpr int kParamOutputsW = 33;    // PFor width w in 0..32
constexpr int kParamCount = 64 * 48 + 64 + 64 * 64 + 64 + 72 * 64 + 72;  // FP32 parameters of the MLP
void launch_block_features(const unsigned long long* v, uint64_t n, float* feats, cudaStream_t st);
// Exhaustive (w, k) search per block; `only` (may be null) restricts it to flagged blocks.
void launch_block_search(const unsigned long long* v, uint64_t n, const uint8_t* only, uint8_t* w, uint8_t* k,
                         uint32_t* cost, cudaStream_t st);
void launch_block_cost(const unsigned long long* v, uint64_t n, const uint8_t* w, const uint8_t* k, uint32_t* cost,
                       cudaStream_t st);
void launch_block_offsets(const uint32_t* cost, uint64_t nblk, unsigned long long* offs, unsigned long long* total,
                          cudaStream_t st);
void launch_block_encode(const unsigned long long* v, uint64_t n, const uint8_t* w, const uint8_t* k,
                         const unsigned long long* offs, uint32_t* payload, cudaStream_t st);
void launch_block_decode(const uint32_t* payload, uint64_t payload_bits, uint64_t n, const uint8_t* w,
                         const uint8_t* k, const unsigned long long* offs, unsigned long long* out, uint32_t* err,
                         cudaStream_t st);
void launch_block_fallback(const float* conf, uint64_t nblk, float thr, uint8_t* flags, unsigned long long* count,
                           cudaStream_t st);
// One (w = 0, k = floor(log2(mean))) pair for every block; sum: device double, zeroed.
void launch_block_global(const unsigned long long* v, uint64_t n, double* sum, uint8_t* w, uint8_t* k,
                         cudaStream_t st);
void launch_mlp_forward(const float* prm, const float* feats, uint64_t count, uint8_t* w, uint8_t* k, float* conf,
                        float* logits, cudaStream_t st);
size_t mlp_gather_floats(uint64_t count);
void launch_mlp_train(const float* prm, const float* feats, const uint8_t* wlab, const uint8_t* klab,
                      const uint32_t* idx, uint64_t first, uint64_t count, float scale, float* grad, float* loss,
                      float* gather, cudaStream_t st);
void launch_mlp_adam(float* prm, float* grad, float* m, float* v, float lr, int step, cudaStream_t st);

// zstd frames on the GPU (k_zstd.cu): frame i of src_len[i] bytes at src[i] into dst[i]
// (capacity cap[i]); out_len[i] = content size or < 0 (zstd_dec.cuh error codes).  The
// pointer and size arrays are in device memory; `workspace` holds count * zstd_workspace_bytes().
size_t zstd_workspace_bytes();
void launch_zstd_frames(const uint8_t* const* src, const uint64_t* src_len, uint8_t* const* dst, const uint64_t* cap,
                        long long* out_len, void* workspace, uint64_t count, cudaStream_t st);

}  // namespace dev
}  // namespace xnyz
