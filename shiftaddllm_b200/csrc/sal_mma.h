// Internal interface between the C ABI (sal_lutgemm.cu) and the tensor-core product (sal_mma.cu).
#ifndef SAL_MMA_H
#define SAL_MMA_H

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>

#include <shared_mutex>

#include "sal_lutgemm.h"

namespace sal_mma {

constexpr int MAX_ROWS = 4096;   // activation rows of one call

// Layout of the multipliers.  ROW: fp16 [num_groups][q][N], a group is K / num_groups input features.  BLOCK_F16 / BLOCK_U16:
// [K/8][q][num_groups], a group is N / num_groups output columns (fp16, or three 3-bit exponents in 16 bits).
enum AlphaLayout { ROW = 0, BLOCK_F16 = 1, BLOCK_U16 = 2 };

struct Problem {
    alignas(64) CUtensorMap tmap;   // packed planes as [K/32 words][q planes][N columns], box [4][q][128]
    CUtensorMap xmap;               // activations as [M rows][K features] fp16, box [mpad][64], 128-byte swizzle
    CUtensorMap smap;               // scales as fp16 rows (see build), if they are fetched by TMA
    const unsigned *bw;
    const unsigned short *alpha;
    const unsigned short *bias;
    const unsigned short *x;
    unsigned short *y;
    int K, N;
    int run;          // ROW: words whose sum the table kernels multiply by a scale at a time
    int s_tx;         // bytes of scales per unit by TMA
    int ku;           // 128-feature units of K
    int unit_begin;   // first unit of the problem in the launch's unit sequence
    int tile_begin;   // first output tile
    int ntiles;       // column tiles x row tiles
    int gw;           // ROW: 32-feature words per group
    int gshift;       // ROW: log2(gw), -1 if it is no power of two
    int ngroups;      // ROW: groups along K; BLOCK: groups along N
    int gs;           // BLOCK: columns per group
};

struct Params {
    Problem p[SAL_MAX_GROUP];
    int count;
    int M;            // activation rows
    int mtiles;       // row tiles
    int mt;           // rows per row tile
    int mpad;         // rows per row tile, rounded up to the 16 of an instruction
    int total_units;
    int whole_tiles;  // one CTA per output tile (no scratch buffer), else equal runs of units per CTA
    int accumulate;
    int layout;
    int use_tma;      // planes fetched by TMA (else 4-byte asynchronous copies)
    int tma_scales;   // scales fetched by TMA
    int s_pitch;      // bytes of a row of scales in the ring
    int w_stages, a_stages, x_units;
    int s_bytes;      // scales of a unit in the ring
    int *status;
    unsigned *counters;   // one per output tile
    float *partials;      // [2 x CTAs][mt][128]
};

struct Built {
    Params P;
    int q, ctas, smem;
    size_t ws_need;          // scratch bytes for arrival counters and partial sums (0: none)
    size_t act_bytes;        // further scratch for silu(x) * x_mul, 0 if not used
    unsigned flags;
    int count;
    const void *gate[SAL_MAX_GROUP], *up[SAL_MAX_GROUP];   // SwiGLU operands (x of the problem is formed in scratch)
};

// Can this product run here at all?
bool eligible(const void *bw, const void *alpha, const void *x, int M, int K, int N, int q, int num_groups, AlphaLayout layout);
// Estimated time in us of a product in one of the BLOCK layouts (see block_tables_us in sal_lutgemm.cu).
double block_us(const sal_problem &problem, AlphaLayout layout, int sms);
// Plans one launch; `ws_bytes` of scratch will be there (0: none).  All problems share M, q and the layout.  `encode`: also encode the
// tensor maps (needs a CUDA context; false for a look at the plan only).
int build(const sal_problem *problems, int count, AlphaLayout layout, unsigned flags, size_t ws_bytes, int sms, Built *out, bool encode = true);
size_t scratch_bytes(const Built &b);   // 0: none
// Scratch with which the split of a product of M rows (without x_mul) follows from its shape alone
size_t full_scratch_bytes(int M);
int launch(const Built &b, void *workspace, size_t ws_bytes, cudaStream_t stream);

}  // namespace sal_mma

// Host threads that share a stream and with it a scratch buffer may enqueue at the same time.  A product that is one launch holds this
// lock shared; one that passes data from launch to launch through the scratch buffer (silu(x) * x_mul of several rows) holds it alone, so
// that no other launch on the same buffer gets in between.  Defined in sal_lutgemm.cu.
std::shared_mutex &sal_scratch_order(const void *workspace);

// Encodes the tensor map of packed planes with the given box (planes x words); defined in sal_lutgemm.cu.
int sal_encode_planes(CUtensorMap *out, const void *bw, int K, int N, int q, int box_cols, int box_planes, int box_words);

// Encodes the tensor map of 16-bit rows [rows][cols] with boxes of box_cols x box_rows, swizzled over 128 bytes or plain.
int sal_encode_rows(CUtensorMap *out, const void *base, int cols, int rows, int box_cols, int box_rows, int swizzle128);

#endif
