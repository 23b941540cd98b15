// vfd_band.h -- axis pass as a banded matrix product on the tensor cores
// (vfd_band.cu), and the per-axis operators it applies.
//
// One substep of a separable world is B_z B_y B_x: per axis, mask (the
// padding rule's interior), convolve with the axis' taps, crop.  The three
// operators act on different axes and commute, so m substeps are
// B_z^m B_y^m B_x^m: three passes over the field instead of 3 m.  B^m is a
// banded n x n matrix, Toeplitz away from the line's ends; it is computed in
// FP64 (its tails beyond a half-width H, whose sum is below 1e-8, are
// moved to H, keeping sum and variance) and applied in blocks of 64 outputs.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "vfd_axis.cuh"

namespace vfd {

constexpr int BD_LINES = 128;   // lines per tile (the M of the tensor-core product, one TMEM lane each)
constexpr int BD_BLK = 64;      // positions per block (inputs and outputs)
constexpr int BD_HMAX = 56;     // largest half-width of B^m (two images and two stages fit shared memory)
constexpr int BD_MMAX = 16;     // most substeps folded into one operator
constexpr int BD_NBMAX = 33;    // blocks of the longest line (2047 positions, plus the half-width)
constexpr int BD_STEP_BYTES = 3 * BD_BLK * 16 * 2;  // one k-step (16 positions) of an image: 3 bf16 parts

// One (field, axis) pass.  Lines are numbered through the whole field:
// x pass: line l is row l (position stride 1); y / z pass: line l sits at
// (l / n0) * outer_stride + l % n0.
struct alignas(16) BandJob {
    float *data;
    double *mass;
    const unsigned char *img;  // this axis' weight images (BandAxis)
    const CUtensorMap *map;    // tensor map of the input blocks, or NULL (copied by cp.async)
    const float *rho;          // row sums of the images, 64 each: over the window's first input block, its first two, all
    const float *fn;           // functional weights by input position: alpha[nin * 64], then lambda[nin * 64]
    const float *lw1, *lw2;    // line weights: x pass alpha_y, alpha_z; y pass (lw2) alpha_z
    const float *aff[3];       // affine rows X_j, Y_j, Z_j (z pass, naff > 0), row stride affs[a]
    const float *affc;         // their coefficients
    int *gave_up;              // set where a wait gave up (the world's)
    int64_t outer_stride, pos_stride;
    unsigned long long plain;  // bit k: input block k has alpha = 1 and lambda = 0 everywhere
    int affs[3];
    int naff;
    int n, n0, nlines, ntiles, tile0;
    int H, ksteps, nb, nin;    // half-width, k-steps of an image, output and input blocks
    int b0, b1;                // output blocks b0 .. b1 - 1 see no boundary: they share image b0
    unsigned char kind;        // PassKind
    bool vec;                  // 16-byte accesses apply
    bool mask;                 // x pass: apply the padding rule
    bool sums;                 // form the accounting (a launch may turn it off for all)
    float b, keep, fscale;     // fscale: factor folded into the operator (x pass: keep^(m-1), z pass: keep, y pass: 1)
    int nx, ny;
    int box_lo[3], box_hi[3];
    // image of output block b
    __host__ __device__ int image(int b) const { return b < b0 ? b : b < b1 ? b0 : b - (b1 > b0 ? b1 - b0 - 1 : 0); }
};
static_assert(sizeof(BandJob) % 16 == 0, "BandJob is copied in 16-byte pieces");

// What the set-up kernels need of a (field, axis) operator.
struct BandAxis {
    const double *taps;     // 2 r + 1
    unsigned char *img;     // nimg images of ksteps * BD_STEP_BYTES
    float *rho;             // row sums of the images (as BandJob::rho)
    float *fn;              // alpha, lambda (as BandJob::fn)
    float *aff;             // naff rows of affs floats (X_1 .. X_naff)
    double *dots;           // [3][BD_MMAX]: sum M X_j, sum lambda_0 X_j, sum X_j
    double scale, fscale;   // folded into the images / the functional weights
    int n, r, m, H, ksteps, nin, lo, hi, nimg, affs, naff;
    int blk[BD_NBMAX];      // output block of each image
};

// Per field: the accounting block a tick starts from (zero, or what the
// affine part of the padding rule adds).
struct BandInit {
    const double *dots[3];
    double *out;            // MS_COUNT doubles
    float *affc;            // coefficients of the affine rows, j = 1 .. naff
    double c, keep;         // (keep - 1) b, and keep
    int naff;
};

// Encodes the tensor map of job j's input blocks (x pass: boxes of 32
// positions x 128 rows; y / z pass: of 32 lines x 64 positions); false if the
// layout does not allow it (rows or planes not 16-byte aligned, y-pass tiles
// whose 32-line runs would cross rows).
bool band_encode_map(const BandJob &j, int nz, CUtensorMap *m);

// out[m - 1]: the half-width of the m-fold kernel (taps: 2 r + 1 of FP64) beyond
// which its tails sum to less than 1e-8, rounded up to a multiple of
// 4, for m = 1, 2, ... while it is at most hmax; returns the number of those.
int band_half_widths(const double *taps, int r, int mmax, int hmax, int *out);

// Builds the images and vectors of naxes operators and the nfields
// accounting starts on `st` (device arrays).
cudaError_t launch_band_setup(const BandAxis *axes, int naxes, int max_rows, const BandInit *init, int nfields,
                              cudaStream_t st);

// One pass over tiles tile_begin .. tile_begin + ntiles - 1 of `jobs`, all of
// one axis: tile t belongs to job tjob[t], counted from its tile0.  `geo`
// covers every job.  sums: form the accounting.
struct BandGeom {
    int ksteps = 0;  // largest of the jobs
};
cudaError_t launch_band(const BandJob *jobs, const int *tjob, int tile_begin, int ntiles, int axis,
                        BandGeom geo, bool sums, cudaStream_t st);

// The passes' bounded wait on a barrier that nothing completes: it gives up
// after `limit` cycles, which *gave_up tells as a pass would.
cudaError_t band_wait_probe(long long limit, int *gave_up, cudaStream_t st);

}  // namespace vfd
