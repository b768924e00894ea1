// Non-uniform FFTs on the polar Fourier grids of LaminoCam, FINUFFT semantics:
//   type 1 (iflag +1):  f_k = sum_j c_j exp(+i k.x_j)
//   type 2 (iflag -1):  c_j = sum_k f_k exp(-i k.x_j)
// with modes k in [-floor(N/2), floor((N-1)/2)] in increasing order and x the
// fastest dimension (include/nufft.h:37-95 of the reference).
//
// Non-uniform points are never stored: they are regenerated in FP64 from the
// grid description (polar radius/angle in 2D, rotated detector lattice in 3D)
// wherever a kernel needs them.  Only a permutation that sorts point indices
// by fine-grid bin is kept per (geometry, fine grid).
#pragma once

#include <vector>

#include "lc_fft.hpp"

namespace lc {

// Polar grid description.  2D: x = r cos(theta), y = r sin(theta),
// r_m = (m+1/2) 2pi/nr - pi (include/polar_grid2d.h:50-65).  3D: rows of the
// detector lattice rotated by transpose(Rx(theta) Ry(beta) Rz(gamma))
// (include/polar_grid.h:52-94, include/rotation.h:28-56).
struct PolarPts {
    int dim = 2;
    long M = 0;  // below 2^31 (the bin sort stores point indices as int)
    int ntheta = 0;
    // 2D
    int nr = 0;
    const double2 *cs = nullptr;  // (cos theta, sin theta) per angle
    // 3D
    int nrows = 0, ncols = 0;
    const double *rot = nullptr;  // R00 R01 R10 R11 R20 R21 per angle
    // The lattice of an angle (lat = nr points in 2D, nrows * ncols in 3D) is
    // closed under negation: lattice point l and lat - 1 - l are opposite.  A
    // plan handles one point of each pair, half = ceil(lat / 2) per angle,
    // l < half.  Angles whose lattices hold the same points (axes equal up to
    // sign: theta and theta + 180 degrees of a full turn) share one
    // representative: nrep of them, Mh = nrep * half folded points in all.
    // Members of representative r: mem[moff[r] .. moff[r + 1]), the angle and
    // the flips that map the representative's lattice onto the member's (bit
    // 0: columns, or the radius in 2D; bit 1: rows).
    int lat = 0, half = 0, nrep = 0;
    long Mh = 0;
    const int *moff = nullptr;
    const int2 *mem = nullptr;  // the first member is the representative, unflipped
    const double2 *rcs = nullptr;  // cs and rot of the representatives
    const double *rrot = nullptr;
    // folded point index -> representative (by half) and, in 3D, lattice point -> row (by ncols)
    FastDiv div_angle, div_col;
};

struct PolarGeometry {
    PolarPts pts;
    std::vector<double> theta, gamma, beta;
    std::vector<float> shifts;  // 2 per angle (dx, dy), 3D only
    DevBuf<double2> cs;
    DevBuf<double> rot;
    DevBuf<float2> dshifts;
    DevBuf<int> moff;
    DevBuf<int2> mem;
    DevBuf<double2> rcs;
    DevBuf<double> rrot;
};

void geometry_init_2d(Context &ctx, PolarGeometry &g, const double *theta, int ntheta, int nr);
void geometry_init_3d(Context &ctx, PolarGeometry &g, const double *theta, const double *gamma,
                      const double *beta, const float *shifts, int ntheta, int nrows, int ncols);

// kernel width and shape for a requested tolerance (upsampling factor 2)
int es_width_for_tol(double tol);
double es_beta_for_width(int w);

// Pointwise handling of the non-uniform values inside spread / interp.
enum PtMode {
    PT_PLAIN = 0,   // values used as given
    PT_MASK = 1,    // multiply by the 3D |q|<=pi mask w_j
    PT_SHIFT = 2,   // 3D: mask and exp(-i(qX dx + qY dy)) per projection
};

// NUFFT plan for one geometry and one mode box (x, y[, z] = n3, n2[, n1]).
class NufftPlan {
  public:
    NufftPlan(Context &ctx, const PolarGeometry &g, const int modes[3], double tol);
    // device memory of a plan over ntheta lattices of lat points and of its
    // buffers for nvol volumes (an upper bound: angles may share their points)
    static size_t device_bytes(int dim, const long modes[3], double tol, long ntheta, long lat, long nvol);
    // type 1: c [nvol][M] complex -> out real [nvol][n1][n2][n3] = Re(f) * scale.
    // herm: the values at opposite lattice points are conjugates; only lattice
    // points below half are read.  (Any plan geometry; see fold_values_kernel.)
    void type1_real(Context &ctx, const float2 *c, int nvol, float *out, float scale,
                    PtMode mode, bool herm = false);
    // type 2: real in [nvol][...modes] -> c [nvol][M].  keep > 0: only lattice
    // points below it (and at least half) are stored, and the caller takes the
    // others as their conjugates (see expand_values_kernel for the band limit).
    void type2_real(Context &ctx, const float *in, int nvol, float2 *c, PtMode mode, int keep = 0);

    int dim() const { return dim_; }
    long M() const { return pts_.M; }
    const int *nf() const { return nf_; }
    int width() const { return w_; }

  private:
    void sort_points(Context &ctx);
    void spread(Context &ctx, const float2 *c, int nvol, float2 *grid, PtMode mode, bool herm);
    void interp(Context &ctx, const float2 *grid, int nvol, float2 *c, PtMode mode, int keep);

    int dim_;
    PolarPts pts_;
    const float2 *shifts_ = nullptr;
    int modes_[3];
    int nf_[3];
    int w_;
    double beta_;
    int ny_, ylo_;  // fine-grid rows kept: ny_ rows from row -ylo_ (mod nf_[1])
    int bs_[3];
    int nb_[3];
    DevBuf<float> corr_[3];
    DevBuf<float> corr_xy_;  // corr_y (x) corr_x, 3D type 2
    DevBuf<int> perm_;
    DevBuf<unsigned short> corner_;  // per sorted point: footprint corner in its bin's tile, band flag
    DevBuf<float2> vals_;            // folded values, [nvol][Mh]
    DevBuf<int4> subs_;
    int nsub_ = 0;
    int maxsub_ = 1024;  // most points of one spreading subproblem
    long kmax_ = 1;      // bound on the footprints that cover one fine-grid cell
    DevBuf<float2> grid_, h1_, h2_;
    DevBuf<long long> fix_;  // 64-bit fixed-point fine grid of the spreading (re, im)
    DevBuf<int> mbits_;      // bound on the spread values (float bits)
    DevBuf<int> kbin_;       // per bin: bound on the summed weights over one tile cell (float bits)
    DevBuf<int> binm_;       // per bin and chunk of volumes: bound on its spread values (float bits), per call
};

}  // namespace lc
