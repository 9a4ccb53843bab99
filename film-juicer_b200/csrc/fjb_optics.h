// fjb_optics.h -- parameter blocks of the separable optics passes (scatter/halation).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <string>

#include "../../include/juicer_cuda_api.h"
#include "fjb_line_pairs.cuh"

namespace fjb {

// Gaussian operator kinds, numbered as FJ_HALATION_* in the C-ABI.
enum GaussKind : int { kGaussIdentity = 0, kGaussFir = 1, kGaussYvv = 2, kGaussYvvFactored = 3 };

constexpr int kOpticMaxGauss = 5;
constexpr int kOpticMaxFirRadius = 9;

constexpr int kOpticSeg = 64; // segment length of the block-parallel recursions

struct OpticGauss {
    int kind;
    int radius;   // FIR only
    float w[19];  // FIR weights, w[radius] is the centre tap
    float yvv[4]; // legacy: B, B1, B2, B3; factored: h, g, t, 0
    // recursive kinds, the zero-input state maps (row-major 3x3) that the pass's form needs:
    // over a piece of a row and of a column and their powers, or over kOpticSeg steps
    lp::LineMaps row_maps, col_maps;
    double seg[9];
};

enum OpticMode : int { kOpticScatter = 0, kOpticBounce = 1 };

// One channel plane and the Gaussians evaluated on it in one sweep.
struct OpticJob {
    float* src;        // carrier plane, read, then overwritten by the combination
    long long stride;  // floats per row of src
    float* temp[kOpticMaxGauss]; // row-filtered planes, width floats per row
    int count;         // Gaussians in g[]
    OpticGauss g[kOpticMaxGauss];
    float coef[kOpticMaxGauss]; // tail amplitudes (scatter) or bounce weights (bounce)
    int mode;          // OpticMode
    int tail_count;    // scatter: g[0..tail_count) are tails, g[tail_count] is the core
    float tail_weight; // scatter only
    float amount;      // scatter amount, or bounce total strength
    int renormalize;   // bounce only
    // one warp per pair of lines: the combination as weights of the carrier and of each
    // Gaussian, and the plane the column launch adds its Gaussians to (null: the carrier
    // times its weight)
    float carrier_weight;
    float weight[kOpticMaxGauss];
    float* base;
};

struct OpticPass {
    int width, height, jobs;
    OpticJob job[3];
    // block-parallel recursion buffers: 3 floats of segment state per (job, Gaussian,
    // line, segment) and two per-line edge values per (job, Gaussian, line)
    float* carry;
    float* edge_a;
    float* edge_b;
    int lines_max, segs_max;
    // the whole scratch of the stage; one warp per pair of lines: the pairs a row and a column
    // CTA hold, the recursions a column CTA holds at once, the rows and column CTAs between a
    // CTA and the one after it, and whether every job has a plane `base`
    float* scratch;
    size_t scratch_floats;
    int row_pairs, col_pairs, recursions, rows_ahead, cols_ahead;
    bool taps_for_all;
};

cudaError_t launch_optic_pass(OpticPass& P, cudaStream_t stream);

// One warp per pair of lines (fjb_halation_lines.cu): false when the pass's lines or planes are
// out of its range; true lays the pass out for launch_optic_lines.
bool optic_lines_plan(OpticPass& P);
cudaError_t launch_optic_lines(OpticPass& P, cudaStream_t stream);

// One zero-input step of a recursive Gaussian's state (row-major 3x3).
void optic_step_map(const OpticGauss& g, double m[9]);

// Segments of the block-parallel recursions along a line of n samples.
int optic_segments(int n);

// Scratch floats needed by scatter_halation for a width x height frame.
size_t halation_scratch_floats(int width, int height);

// Runs scatter then back-reflection on the three carrier planes (R, G, B order of the
// descriptor's channels). `scratch` holds halation_scratch_floats() floats.
bool scatter_halation(const FjScatterHalation& d, float* planes_rgb[3], long long stride, int width, int height,
                      float* scratch, cudaStream_t stream, std::string& why, cudaError_t& err);

} // namespace fjb
