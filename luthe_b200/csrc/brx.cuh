// Tensor-core blind rotation (brx.cu): sizes and launch wrappers.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include "kernels.cuh"

namespace luthe {
namespace brx {

constexpr int PK = 64;                       // evaluation points of Y = X^32 (Y^64 = -1): 32 and their inverses
constexpr int PH = PK / 2;
constexpr int XN = 32;                       // coefficients left at each point
constexpr int TILE = 128;                    // ciphertexts per product tile (MMA rows)
constexpr int CORES = 2 * XN - 2;            // core matrices of one Toeplitz block
constexpr size_t BLOCK_BYTES = CORES * 128;  // one (point, column, row) block
constexpr size_t STEP_BYTES = PK * 4 * BLOCK_BYTES;
constexpr size_t WF_BYTES = 6 * PH * 8 * PH;  // forward transform weights, 48 KiB
constexpr size_t WI_BYTES = 8 * PH * 8 * PH;  // inverse transform weights, 64 KiB
constexpr size_t WEIGHT_BYTES = WF_BYTES + WI_BYTES + 128 * 8;  // and a table of roots of unity
constexpr size_t TILE_WORDS = (size_t)TILE * 2 * N;  // u64 of one tile's evaluations (4 MiB)
constexpr size_t WAVE = 592;                 // ciphertexts of one launch (two pairs per SM)
constexpr size_t TILES = (WAVE + TILE - 1) / TILE;

struct alignas(64) TensorMap {  // CUtensorMap
    uint64_t opaque[16];
};

// Launches that overlap on the GPU must not share eval, prod, acc and sync.
struct Workspace {
    uint8_t *weights = nullptr;   // [WF][WI][roots]
    uint8_t *bsk = nullptr;       // [n][PK][col][row][BLOCK_BYTES]
    uint64_t *eval = nullptr;     // [TILES][PK][4 atoms][TILE][16] u64: transformed digits
    uint64_t *prod = nullptr;     // [TILES][PK/2][XN][TILE][4] u64: products at pairs of points
    uint64_t *acc = nullptr;      // [TILES * TILE][2][N] u64: accumulators
    uint32_t *sync = nullptr;     // grid-wide progress counters
    TensorMap prod_map;           // of prod
    const unsigned long long *polls = nullptr;  // device-wide bound on slab waits
};
constexpr size_t EVAL_WORDS = TILES * TILE_WORDS, PROD_WORDS = EVAL_WORDS, ACC_WORDS = EVAL_WORDS;
constexpr size_t SYNC_BYTES = 128 * (1 + 2 * TILES);
constexpr size_t BUFFER_BYTES = (EVAL_WORDS + PROD_WORDS + ACC_WORDS) * 8 + SYNC_BYTES;  // 63 MB: what a launch writes

// is the stream confined to some of the device's SMs (a green context's)?  launch() must not be called on one
bool limited_stream(cudaStream_t s);
void build_weights(uint8_t *host /* WEIGHT_BYTES */);
cudaError_t set_attributes();
cudaError_t make_prod_map(Workspace &ws);
// expand the standard-domain BSK ([n][row][col][N], values < p) into ws.bsk
cudaError_t launch_expand(const uint64_t *d_std_p, const Workspace &ws, uint32_t n, cudaStream_t s);
// blind rotation and sample extract of B <= WAVE ciphertexts (one launch)
cudaError_t launch(const Workspace &ws, int nsm, const uint32_t *d_lwe2N, const uint64_t *d_luts,
                   const uint32_t *d_lut_id, uint32_t nlut, uint64_t *d_out, size_t B, uint32_t n, uint32_t *d_err,
                   cudaStream_t s, uint32_t mlk, uint32_t pbs_bw, uint32_t tie_rule);

}  // namespace brx
}  // namespace luthe
