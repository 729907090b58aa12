// Short-range erfc tree walk (crates/gadget-ng-treepm/src/short_range.rs).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tree.cuh"

namespace tpm {

constexpr int POLY_DEGREE = 10;
// P with erfc(x) = 2^P(x) on [0, x_max]: coefficients of powers of x, and the
// end of the range on which it may be used: at most x_far, and 0 when x_max
// itself is beyond what a polynomial of this degree fits.
struct ErfcPoly {
  double coef[POLY_DEGREE + 1];
  double end;
};
ErfcPoly erfc_poly(double x_max, double x_far);

struct WalkArgs {
  int64_t n, n_int;
  // particles, sorted order
  const uint32_t* qx;
  const uint32_t* qy;
  const uint32_t* qz;
  const float* massf;
  // octree
  const WalkNode* recs;  // walk records, children contiguous
  const uint4* walk;  // internal nodes: fixed-point COM + float mass bits
  const uint8_t* depth;
  const uint32_t* slots;  // eight child slots per internal node
  const double* o_com;
  const uint8_t* leaf_depth;
  // groups
  const uint32_t* gfirst;
  const uint32_t* gsize;
  const uint32_t* ngroups;  // on the device
  uint32_t* work;
  // geometry (float64 = the reference's decisions; float32 = the fast path)
  double scale, box, rc2, thr, h0;
  int periodic;
  float u_inv;    // 2^-U: quanta -> walk units u = scale * 2^U
  float box_u;    // box side in walk units (2^32 quanta)
  float h0_u;     // root half side in u
  float rc2_lo, rc2_hi;    // per-target ambiguity band around r_cut^2 (u^2): node refinement
  float rc2_mid, rc2_band; // its middle, and half its width (rounded up)
  float prc2_lo, prc2_hi;  // the pair loop's (narrower) band: leaf pairs and monopoles
  float prc2_mid, pband;   // its middle, and half its width (rounded up)
  float grc2_lo, grc2_hi;  // group-level band
  float eps2_u;
  unsigned long long eps2_2;  // two floats: max(eps^2, 1e-30) in u^2 (no quantum squared is as small)
  int poly;       // erfc as 2^P(r): P's coefficients, each as two floats
  unsigned long long poly2[POLY_DEGREE + 1];
  int close;      // exact coordinate differences for pairs near against the group's extent
  float h_term;   // parity: cull half side of the monopoles (all at the terminal depth)
  int term_depth; // the first depth whose half side is below 0.1 r_cut
  float pcx;      // 0.3275911 * scale*2^U / (sqrt(2) r_s)
  float ex2k;     // -(scale*2^U / (sqrt(2) r_s))^2 * log2(e)
  float tiny_u;   // (4 quanta)^2 in u^2
  float out_scale;  // 1/u^2 in physical units
  int accurate;      // extension mode: complete split kernel + opening angle
  float theta2;      // opening angle squared (accurate mode)
  float gkc;         // (2/sqrt(pi)) * u/(sqrt(2) r_s): the Gaussian term of the split
  int relative;      // accurate mode: relative opening criterion instead of the opening angle
  float rel_k;       // err_tol * u^3 (relative criterion, walk units)
  const uint4* cellq;  // per internal node: fixed-point cell centre, |Q|_F float bits
  // outputs (physical, per unit G), sorted order
  float* ax;
  float* ay;
  float* az;
  unsigned long long* stats;  // [0] leaf pairs [1] monopoles [2] evaluated [3] exact fallbacks [4] deferred
  uint32_t* err;
  uint2* deferred;
  uint32_t* ndeferred;
  uint32_t cap_deferred;
  uint32_t* stack;
  uint32_t* pcounts;     // per target (sorted order): leaf pairs, monopoles
  const uint8_t* only;   // nullptr, or: walk only the targets p with only[p] != 0
  int img_depth;         // periodic: nodes shallower than this need the +-L images in the group cull
};

constexpr int WALK_TARGETS = 32;  // targets per warp at most
int walk_group_size(int64_t n);   // targets per walk group in a box of n particles
int walk_blocks_per_sm(bool periodic, bool accurate);
size_t walk_stack_words(int grid);  // the walk's stacks, in 32-bit words
void launch_walk(const WalkArgs& a, int grid, cudaStream_t s);
void launch_deferred(const WalkArgs& a, cudaStream_t s);

}  // namespace tpm
