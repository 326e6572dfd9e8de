// zstd frames decoded on the GPU, one frame per block (zstd_dec.cuh), for callers that hold
// many container frames in device memory: no host round trip.
#include "kernels.h"
#include "zstd_dec.cuh"

namespace xnyz {
namespace dev {

namespace {

struct Workspace : zd::Tables {
    zd::u8* lit;
};

// One frame per block of 128 threads (zd::BlockTeam), the tables in shared memory.  Registers (80) and shared
// memory (35 KB) for six blocks per SM, 888 frames at once; with 96 registers, so five blocks, an earlier
// state took 2.10 ms instead of 1.98.  Bound by latency: the frames with the most sequences (6170 in 28 KB)
// are last, for whom the states' chain takes 160 clocks a sequence and the copies, beside it in other
// warps, about as much.  One warp per frame, whose lanes walked the sequences together, byte loads for the
// bits, tables in global memory and one copy after another took 6.9 ms for 768 frames of 27 KB (81 KB of
// content); this takes 1.4 ms.
__global__ void __launch_bounds__(zd::BlockTeam::size, 6) zstd_frames_kernel(const uint8_t* const* src, const uint64_t* src_len,
                                                                          uint8_t* const* dst, const uint64_t* cap,
                                                                          long long* out_len, uint8_t* literals) {
    __shared__ Workspace ws;
    __shared__ int slot;
    const uint64_t f = blockIdx.x;
    const zd::BlockTeam team{(int)threadIdx.x, &slot};
    if (team.rank == 0) ws.lit = literals + f * (zd::kMaxBlock + 32);
    __syncthreads();
    const long long r = zd::decode_frame(src[f], src_len[f], dst[f], cap[f], ws, team);
    if (team.rank == 0) out_len[f] = r;
}

}  // namespace

size_t zstd_workspace_bytes() { return zd::kMaxBlock + 32; }

void launch_zstd_frames(const uint8_t* const* src, const uint64_t* src_len, uint8_t* const* dst, const uint64_t* cap,
                        long long* out_len, void* workspace, uint64_t count, cudaStream_t st) {
    if (!count) return;
    zstd_frames_kernel<<<(unsigned)count, zd::BlockTeam::size, 0, st>>>(src, src_len, dst, cap, out_len, static_cast<uint8_t*>(workspace));
}

}  // namespace dev
}  // namespace xnyz
