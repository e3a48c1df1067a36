// hj_host.h -- host-side table builders (hj_host.cpp), not part of the ABI.
#pragma once

#include <cstdint>

#include "../../include/haissinski_gpu.h"

namespace hj {
double host_wake_function(double c, const hj_wake& w);
double host_delta(double x, double sigma);
void host_wake_tables(const double* centers, int64_t B, const hj_wake& w, double* W,
                      double* lam);
// The centre w(2k+1-B)/B of bin k, correctly rounded (hj_make_grid).
double host_center(double w, int64_t k, int64_t B);
// Half width of the grid of a bunch of initial length sigma_z0 and its edge step.
double host_half_width(double sigma_z0, double half_width_sigmas);
double host_edge_step(double w, int64_t B);
// The wake of uniform centres as a geometric sequence: J = the last bin whose
// centre is <= 0, W[J-d] = Re(A σ^d) with σ = exp(-step (1/cτ + i s)), and pw[k] =
// σ^{2^k}, k < npw, tau = σ^{J+1}; complex values as (re, im) pairs, in extended
// precision and rounded once.
void host_wake_powers(const hj_wake& w, double cJ, double step, int64_t J, double A[2],
                      double tau[2], double (*pw)[2], int npw);
// Whether the B centres are uniform to rounding with a positive step and reach
// <= 0, i.e. the wake table is that sequence; J and the step when so.
bool host_uniform_centers(const double* centers, int64_t B, int64_t* J, double* step);
// Whether the interpolation cells of a caller's grid (between its centres) start half a
// bin off its histogram's bins (between its edges) throughout, to rounding: then the
// halves of a cell are those of two neighbouring bins.
bool host_cells_halve_bins(const hj_grid& g);
// Cell coordinate v = z inv + off of the kick table (cell j between centres j-1 and j):
// from the edges where the cells halve the bins, else from the centres c1 and cB.
void host_kick_cells(bool halves, int64_t B, double e0, double inv_e, double c1, double cB,
                     double inv_c, double* inv, double* off);
// Particle factor of the wake current (src/evolution.jl:373-384).
double host_particle_factor(int64_t n, double population);
void host_twiddles(int64_t P, double* tw_interleaved);
// cos and sin of 2π m / M, m < M, each as a sum of two doubles: (cos hi, lo, sin hi, lo).
void host_rf_unit(int M, double (*unit)[4]);
// sin and cos of phi likewise: (sin hi, lo, cos hi, lo).
void host_sincos(double phi, double out[4]);
// Tables of the device's Float64 normals: a 2048-layer ziggurat for the
// density f(x) = exp(-x²/2), x >= 0 (G. Marsaglia and W. W. Tsang, "The
// Ziggurat Method for Generating Random Variables", J. Stat. Softw. 5(8),
// 2000), as hj_device.cuh (zig_fast, zig_slow) samples it.  Layer 0 is the
// base: the rectangle [0, r) x [0, f(r)) plus the tail x >= r, of area v;
// layer i >= 1 is the rectangle [0, X_i) x [f(X_i), f(X_{i+1})), also of
// area v, with X_1 = r, X_2048 = 0 and X_0 = v / f(r).
constexpr int kZigLayers = 2048;
struct NormalTables {
  // (X_i, D_i): layer i's width and its fast-acceptance bound D_i = 1 + K_i 2^-52,
  // K_i = ceil(2^52 X_{i+1} / X_i): a draw U = m 2^-52 of layer i with
  // 1 + m 2^-52 < D_i lies under the curve whatever its height.
  double xd[kZigLayers][2];
  double f[kZigLayers + 1];   // f(X_i), f(X_2048) = 1: the wedge tests
  double r;                   // X_1: where the tail begins
  double v;                   // the common area of the layers
};
// Solves for r in extended precision (bisection on the layer recursion
// X_{i+1} = sqrt(-2 ln(f(X_i) + v / X_i)) until X_2048 = 0) and fills the
// tables, each entry rounded once.
void host_normal_tables(NormalTables* t);
}  // namespace hj
