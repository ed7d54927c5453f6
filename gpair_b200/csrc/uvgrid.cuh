// uvgrid.cuh -- the uv-grid plan of a context (uvgrid.cu).
#pragma once

#include "gpair_internal.cuh"

#define UG_W 8  // window width in grid points
#define UG_OVERSAMPLING 2.0  // grid points per cycle and image width (2.5 and 3 measured no more accurate: FP32 rounding remains)
#define UG_MAX_SPLITS 8  // partial sums of the x contraction

// A problem takes the grid when the image is at least UG_MIN_WIDTH wide, its direct work 2 N^2 nuv is at
// least UG_MIN_WORK_* of the precision mode and UG_GRID_RATIO times the grid's own contractions, and the
// coverage is not too wide for the mode (UG_WIDE_RATIO_*).
// UG_MIN_WIDTH: on narrower images hundreds of uv points share a grid point, and its FP32 rounding no
// longer averages out of the gradient (2e-7 to 4e-7 at 55 to 67 pixels, the direct sums 1e-7).
// UG_MIN_WORK_FP32: where the CUDA-core contractions start to cost more than the grid's fixed launches
// (an objective with its gradient + eight trials, directly and through the grid: 147^2 x 1,904 uv 82 + 100 us, 77 + 42;
// 128^2 x 1,300 67 + 61, 71 + 38; 128^2 x 960, objective and gradient: 59, 66).
// UG_MIN_WORK_TC, _F8: not where the times cross (128^2 x 1,300 uv points, below 960 at 256^2), but how far the modes
// keep the results of their direct sums: those sums' rounding, 1e-6 to 1e-5 of the gradient and largest with E4M3 cross terms, is a
// hundred times the grid's, and a CG run a few iterations on differs by up to 5e-5 with it. What that costs (the same two
// times): split-f16 128^2 x 4,480 79 + 42, 76 + 42; 192^2 x 6,000 83 + 55, 79 + 47; 256^2 x 960 86 + 39, 78 + 45; x 8,960
// 95 + 71, 79 + 48; split-f16/E4M3 256^2 x 21,120 118 + 100, 79 + 48; x 30,000 132 + 129, 82 + 49. From 1.2e9 to 4e9
// split-f16 is therefore the faster of the two.
// UG_WIDE_RATIO_TC (SPLIT16), _F8 (SPLIT16F8 and TF32, whose direct forwards cost two thirds): on a wide
// coverage the grid's y contractions, FP64 on nbx (2 J + 1) grid points, are slower than the tensor cores' direct sums,
// which the ratio above does not see. One objective with its gradient + eight trials, direct and through the grid, split-f16:
// half a cycle per pixel each way, 1024^2 x 8,924 uv 335 + 626 us and 3,880 + 6,060, 512^2 x 8,412 112 + 127 and 613 + 722,
// x 134,607 717 + 1,938 and 729 + 954; a quarter of a cycle, 512^2 x 12,907 131 + 183 and 224 + 252, x 51,631
// 311 + 749 and 232 + 315. At the lines an objective with its gradient and two batches of eight trials cost the same within a
// fifth; an ordinary coverage (1024^2: 60 x 119 grid points) is far above them. The direct sums are less accurate there, within
// the modes' bounds (515^2 x 9,001 over the whole plane, adjoint of given weights: 7e-6 against 1.5e-7). FP32 and
// TF32X3 have no such line, because that difference passes their bounds: TF32X3 1.4e-5 directly (bound 1e-5), FP32 gradient
// 1.6e-5 directly and 1.8e-6 through the grid.
#define UG_WIDE_RATIO_TC 300.0
#define UG_WIDE_RATIO_F8 450.0
#define UG_MIN_WIDTH 96
#define UG_MIN_WORK_FP32 4e7
#define UG_MIN_WORK_TC 1.2e9
#define UG_MIN_WORK_F8 4e9
#define UG_GRID_RATIO 4.0

struct UgState {
    int N, H;            // image width, folded width (N + 1) / 2
    int jxf, nbx, J;     // grid columns jxf .. jxf + nbx - 1, rows -J .. J
    int cells, nchunk;   // nbx (2 J + 1); runs of at most 32 uv points of one cell
    int ldT;             // floats per row of T
    void *mem;           // what the arrays up to S lie in
    // uv points sorted by the cell of their first window point
    int *src;            // [nuv] uv index, bit 31: conjugated
    int *base;           // [nuv] cell
    float *wts;          // [nuv][2 UG_W] window weights along x, then y
    float2 *phase;       // [nuv] e^{2 pi i (a - b)(N-1)/2}
    int2 *chunk;         // [nchunk] (first point, points)
    int *cst;            // [cells + 1] first run of every cell
    float2 *ftab, *ctab; // grid twiddles [nbx][H], [H][J + 1] (k_ug_tables)
    double *invphi;      // [H] 1 / window transform
    // the x contraction's sums, on the CUDA cores [0] and on the tensor cores [1]: [splits][N][ldT] of one image, where a
    // mode has taken them (t_mem: their own allocation, if any)
    float *T[2];
    void *t_mem[2];
    float2 *grid;        // [cells] G
    float2 *patch;       // [nchunk][64]
    float2 *cgrid;       // [cells] C
    float2 *S;           // [N][nbx]
    // batched trials
    float *Tb[2];        // [splits][GP_NTR rows per image][ldT], likewise
    float2 *gridb;       // [cells][GP_NTR]
    int splits, splitsb; // partial sums of the last CUDA-core x contraction
};

// Partial sums of the tensor cores' x contraction at most (TC_GRID_PRODUCTS products each)
static inline int ug_tc_splits(int N) { return gp_cdiv(N, 128) < UG_MAX_SPLITS ? gp_cdiv(N, 128) : UG_MAX_SPLITS; }
