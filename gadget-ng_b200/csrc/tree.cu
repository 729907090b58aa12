// Octree construction on the device.
//
// The reference builds its octree by inserting particles one at a time
// (crates/gadget-ng-tree/src/octree.rs:474-540): one particle per leaf, all
// eight children created on each split, octant chosen by `p >= centre`
// comparisons against float64 child centres (octant_of :423-435,
// child_center :447-465).  The resulting node set does not depend on the
// insertion order: a cell is internal iff it holds two or more particles.
// So the device computes, per particle, the exact sequence of octant choices
// the insertion would make (same float64 centres, same comparisons), sorts by
// that path key, and reads the nodes off the numbers of octant levels that
// neighbours in the sorted order share.  Mass, centre of mass and quadrupole are then
// aggregated bottom-up in float64 with the reference's operation order
// (aggregate :547-629), so they are bit-identical to the reference's nodes.
#include "common.cuh"
#include "scan.cuh"
#include "tree.cuh"

namespace tpm {
namespace {

constexpr double F64_EPSILON = 2.220446049250313e-16;

// ---------------------------------------------------------------------------
// bounding box and root cube
// ---------------------------------------------------------------------------
// Seeds the min/max words on the stream (no host copy, so nothing pageable is
// read and the sequence stays stream-ordered).
__global__ void k_bbox_init(uint32_t* __restrict__ out) {
  if (threadIdx.x < 6) out[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
}

__global__ void k_bbox(const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                       const uint32_t* __restrict__ qz, int64_t n, uint32_t* __restrict__ out) {
  uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t a = qx[i], b = qy[i], c = qz[i];
    mn[0] = min(mn[0], a); mx[0] = max(mx[0], a);
    mn[1] = min(mn[1], b); mx[1] = max(mx[1], b);
    mn[2] = min(mn[2], c); mx[2] = max(mx[2], c);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    uint32_t a = __reduce_min_sync(0xffffffffu, mn[d]);
    uint32_t b = __reduce_max_sync(0xffffffffu, mx[d]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&out[d], a);
      atomicMax(&out[3 + d], b);
    }
  }
}

// bounding_cube (octree.rs:1306-1332) and the Hilbert box (sfc.rs:187-204,
// with the extent from SfcDecomposition::build_with_kind, :250-280).
__global__ void k_root(const uint32_t* __restrict__ bb, double scale, TreeParams* __restrict__ prm) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double mn[3], mx[3];
  for (int d = 0; d < 3; ++d) {
    mn[d] = decode(bb[d], scale);
    mx[d] = decode(bb[3 + d], scale);
    prm->qmin[d] = bb[d];
    prm->qmax[d] = bb[3 + d];
  }
  double hx = dmul(dsub(mx[0], mn[0]), 0.5), hy = dmul(dsub(mx[1], mn[1]), 0.5), hz = dmul(dsub(mx[2], mn[2]), 0.5);
  for (int d = 0; d < 3; ++d) prm->center[d] = dmul(0.5, dadd(mn[d], mx[d]));
  double half = fmax(fmax(hx, hy), hz);
  double pad = fmax(dmul(half, 1e-6), 1e-12);
  prm->half = dadd(half, pad);
  for (int d = 0; d < 3; ++d) {
    prm->hlo[d] = mn[d];
    prm->hlen[d] = fmax(dsub(mx[d], mn[d]), F64_EPSILON);
  }
}

// ---------------------------------------------------------------------------
// octant-path keys
// ---------------------------------------------------------------------------
// 21 octant levels of the reference's insertion octree from the cell state
// (centre, half side) onward: the digit is the octant of the particle against
// the centre, then child_center moves the centre by +/- half/2 per axis, all
// in float64 as the reference does.  The levels are unrolled so the digit
// shifts are constants.
__device__ __forceinline__ uint64_t octant_word(double x, double y, double z, double& cx, double& cy, double& cz,
                                               double& h) {
  uint64_t key = 0;
#pragma unroll
  for (int l = 1; l <= KEY_LEVELS / 2; ++l) {
    const double q = dmul(h, 0.5);
    const bool ox = x >= cx, oy = y >= cy, oz = z >= cz;
    const uint64_t digit = (uint64_t)ox | ((uint64_t)oy << 1) | ((uint64_t)oz << 2);
    cx = dadd(cx, ox ? q : -q);
    cy = dadd(cy, oy ? q : -q);
    cz = dadd(cz, oz ? q : -q);
    h = q;
    key |= digit << (63 - 3 * l);
  }
  return key;
}

// Levels 1..21 of every particle (the sort key).  Levels 22..42 only
// separate particles that share the first 21 (tie runs), so k_tie_low makes
// them for those alone.
__global__ void k_tree_keys(const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                            const uint32_t* __restrict__ qz, int64_t n, double scale,
                            const TreeParams* __restrict__ prm, uint64_t* __restrict__ key_hi,
                            uint32_t* __restrict__ perm) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = decode(qx[i], scale), y = decode(qy[i], scale), z = decode(qz[i], scale);
  double cx = prm->center[0], cy = prm->center[1], cz = prm->center[2], h = prm->half;
  key_hi[i] = octant_word(x, y, z, cx, cy, cz, h);
  perm[i] = (uint32_t)i;
}

// After the sort: the low word (levels 22..42) of every particle in a run of
// equal high keys, stored by original index for k_fix_ties.
__global__ void k_tie_low(const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                          const uint32_t* __restrict__ qz, int64_t n, double scale,
                          const TreeParams* __restrict__ prm, const uint64_t* __restrict__ hi,
                          const uint32_t* __restrict__ perm, uint64_t* __restrict__ lo_by_index) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t k = hi[i];
  if (!((i > 0 && hi[i - 1] == k) || (i + 1 < n && hi[i + 1] == k))) return;
  const uint32_t j = perm[i];
  const double x = decode(qx[j], scale), y = decode(qy[j], scale), z = decode(qz[j], scale);
  double cx = prm->center[0], cy = prm->center[1], cz = prm->center[2], h = prm->half;
  (void)octant_word(x, y, z, cx, cy, cz, h);
  lo_by_index[j] = octant_word(x, y, z, cx, cy, cz, h);
}

// Runs of equal high keys (particles sharing the first 21 octant levels) are
// ordered by the low key.  Equal full keys mean coincident positions.  A run that
// is too long is left as it is, and the host makes no tree of such keys.
constexpr int MAX_TIE_RUN = 1 << 14;

__global__ void k_fix_ties(int64_t n, const uint64_t* __restrict__ hi, uint32_t* __restrict__ perm,
                           const uint64_t* __restrict__ lo_by_index, uint64_t* __restrict__ lo_sorted,
                           uint32_t* __restrict__ err) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t k = hi[i];
  const bool starts = (i == 0 || hi[i - 1] != k) && (i + 1 < n && hi[i + 1] == k);
  const bool inside = (i > 0 && hi[i - 1] == k);
  if (!starts) {
    if (!inside) lo_sorted[i] = 0;  // a particle alone in its level-21 cell: its low word is never read
    return;
  }
  int64_t e = i + 1;
  while (e + 1 < n && hi[e + 1] == k && e - i < MAX_TIE_RUN) ++e;
  if (e - i >= MAX_TIE_RUN) {
    atomicOr(err, DEV_ERR_TIE_RUN);
    return;
  }
  // insertion sort of perm[i..e] by the low key (stable)
  for (int64_t a = i + 1; a <= e; ++a) {
    uint32_t pa = perm[a];
    uint64_t ka = lo_by_index[pa];
    int64_t b = a - 1;
    while (b >= i && lo_by_index[perm[b]] > ka) {
      perm[b + 1] = perm[b];
      --b;
    }
    perm[b + 1] = pa;
  }
  for (int64_t a = i; a <= e; ++a) {
    lo_sorted[a] = lo_by_index[perm[a]];
    if (a > i && lo_sorted[a] == lo_sorted[a - 1]) atomicOr(err, DEV_ERR_COINCIDENT);
  }
}

__global__ void k_permute(Particles src, Particles dst, int64_t n, const uint32_t* __restrict__ perm) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t j = perm[i];
  dst.qx[i] = src.qx[j];
  dst.qy[i] = src.qy[j];
  dst.qz[i] = src.qz[j];
  dst.vx[i] = src.vx[j];
  dst.vy[i] = src.vy[j];
  dst.vz[i] = src.vz[j];
  dst.mass[i] = src.mass[j];
  dst.massf[i] = src.massf[j];
  dst.id[i] = src.id[j];
}

// ---------------------------------------------------------------------------
// octree nodes from the sorted keys
// ---------------------------------------------------------------------------
// lev[i] = octant levels that particles i - 1 and i share (-1 at both ends).
// The cell of depth d that holds particle i starts there iff lev[i] < d, and
// holds a second particle iff lev[i + 1] >= d: particle i starts the internal
// nodes of depths lev[i] + 1 .. lev[i + 1], one after the other in the node
// order.  So nodes, parents and ranges come from one byte per particle and short
// scans of it, where a binary radix tree over the keys (searched twice per node,
// six words stored per node, then climbed) took 1.46 of the 2.88 ms of the
// build at 256^3.
constexpr int LEV_SCAN = 16;  // neighbours looked at one by one before the search turns to the keys

// Levels shared by two sorted keys.
__device__ __forceinline__ int shared_levels(uint64_t hi_a, uint64_t lo_a, uint64_t hi_b, uint64_t lo_b) {
  const uint64_t x = hi_a ^ hi_b;
  if (x) return (__clzll((long long)x) - 1) / 3;
  const uint64_t y = lo_a ^ lo_b;
  return y ? KEY_LEVELS / 2 + (__clzll((long long)y) - 1) / 3 : KEY_LEVELS;
}

// Do particles i and j lie in the same cell of depth d (1 .. KEY_LEVELS)?
__device__ __forceinline__ bool same_cell(const uint64_t* __restrict__ hi, const uint64_t* __restrict__ lo,
                                          uint64_t hi_i, uint64_t lo_i, int64_t j, int d) {
  const uint64_t x = hi_i ^ __ldg(&hi[j]);
  if (d <= KEY_LEVELS / 2) return (x >> (63 - 3 * d)) == 0;
  return x == 0 && ((lo_i ^ __ldg(&lo[j])) >> (63 - 3 * (d - KEY_LEVELS / 2))) == 0;
}

// Also counts the nodes of each depth (hist), so that the host learns the
// levels' sizes together with the number of nodes.
__global__ void k_levels(int64_t n, const uint64_t* __restrict__ hi, const uint64_t* __restrict__ lo,
                         int8_t* __restrict__ lev, uint32_t* __restrict__ cnt, uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[DEPTH_BINS];
  if (threadIdx.x < DEPTH_BINS) sh[threadIdx.x] = 0u;
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) {
    const uint64_t h = hi[i], l = lo[i];
    const int before = i > 0 ? shared_levels(hi[i - 1], lo[i - 1], h, l) : -1;
    const int after = i + 1 < n ? shared_levels(h, l, hi[i + 1], lo[i + 1]) : -1;
    lev[i] = (int8_t)before;
    if (i + 1 == n) lev[n] = -1;
    cnt[i] = after > before ? (uint32_t)(after - before) : 0u;
    for (int d = before + 1; d <= after; ++d) atomicAdd(&sh[d], 1u);
  }
  __syncthreads();
  if (threadIdx.x < DEPTH_BINS && sh[threadIdx.x]) atomicAdd(&hist[threadIdx.x], sh[threadIdx.x]);
}

// hist -> exclusive offsets (DEPTH_BINS + 1) and cursors; one warp
__global__ void k_depth_offsets(uint32_t* tab) {
  uint32_t* hist = tab;
  uint32_t* off = tab + DEPTH_BINS;
  uint32_t* cur = tab + 2 * DEPTH_BINS + 1;
  if (threadIdx.x == 0) {
    uint32_t acc = 0;
    for (int d = 0; d < DEPTH_BINS; ++d) {
      off[d] = acc;
      cur[d] = acc;
      acc += hist[d];
    }
    off[DEPTH_BINS] = acc;
  }
}

__device__ __forceinline__ uint32_t digit_at(uint64_t hi, uint64_t lo, int depth) {
  // octant digit chosen at the split of the node at depth-1 (depth >= 1)
  return depth <= 21 ? (uint32_t)((hi >> (63 - 3 * depth)) & 7u) : (uint32_t)((lo >> (63 - 3 * (depth - 21))) & 7u);
}

// Per particle: the nodes that start there, their ranges and parents, its leaf,
// and the child slots of all of them.
__global__ void k_oct_nodes(int64_t n, int64_t n_int, const int8_t* __restrict__ lev, const uint64_t* __restrict__ hi,
                            const uint64_t* __restrict__ lo, const uint32_t* __restrict__ base,
                            int32_t* __restrict__ o_parent, uint8_t* __restrict__ o_depth,
                            uint32_t* __restrict__ o_first, uint32_t* __restrict__ o_last,
                            uint8_t* __restrict__ leaf_depth, uint32_t* __restrict__ slots,
                            uint32_t* __restrict__ max_depth, uint32_t* __restrict__ cursor,
                            uint32_t* __restrict__ by_depth) {
  // the nodes bucketed by depth for the moments: one reserved range per
  // (block, depth); the order inside a bucket is free
  __shared__ uint32_t here[DEPTH_BINS], start[DEPTH_BINS];
  if (threadIdx.x < DEPTH_BINS) here[threadIdx.x] = 0u;
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n)
    for (int d = lev[i] + 1; d <= lev[i + 1]; ++d) atomicAdd(&here[d], 1u);
  __syncthreads();
  if (threadIdx.x < DEPTH_BINS && here[threadIdx.x]) {
    start[threadIdx.x] = atomicAdd(&cursor[threadIdx.x], here[threadIdx.x]);
    here[threadIdx.x] = 0u;
  }
  __syncthreads();
  uint32_t deep = 0;
  if (i < n) {
    const uint64_t h = hi[i], l = lo[i];
    const int before = lev[i], after = lev[i + 1];
    const uint32_t id0 = base[i];
    // the node of depth `before` that holds the particle: it starts at the
    // nearest earlier particle that shares fewer levels with its predecessor
    int32_t up = -1;
    if (before >= 0) {
      int64_t j = i - 1;
      int scanned = 1;
      while (lev[j] >= before && scanned < LEV_SCAN) {  // (lev[0] = -1 ends it)
        --j;
        ++scanned;
      }
      if (lev[j] >= before) {  // a wide cell: double the step, then halve it
        int64_t in = j, out = -1;
        for (int64_t step = LEV_SCAN; in - step >= 0; step <<= 1) {
          if (!same_cell(hi, lo, h, l, in - step, before)) {
            out = in - step;
            break;
          }
          in -= step;
        }
        while (in - out > 1) {
          const int64_t mid = out + ((in - out) >> 1);
          if (before == 0 || same_cell(hi, lo, h, l, mid, before)) in = mid;
          else out = mid;
        }
        j = in;
      }
      // (in range for keys in order, the only ones that come here)
      const int64_t u = (int64_t)base[j] + (before - lev[j] - 1);
      up = u >= 0 && u < n_int ? (int32_t)u : -1;
    }
    const uint32_t c = after > before ? (uint32_t)(after - before) : 0u;
    int64_t end = i + 2;  // first particle outside the node, deepest node first
    int left = LEV_SCAN;
    for (int d = after; d > before; --d) {
      const uint32_t id = id0 + (uint32_t)(d - before - 1);
      while (left > 0 && lev[end] >= d) {  // (lev[n] = -1 ends it)
        ++end;
        --left;
      }
      if (lev[end] >= d) {
        int64_t in = end, out = n;
        for (int64_t step = LEV_SCAN; in + step < n; step <<= 1) {
          if (d > 0 && !same_cell(hi, lo, h, l, in + step, d)) {
            out = in + step;
            break;
          }
          in += step;
        }
        while (out - in > 1) {
          const int64_t mid = in + ((out - in) >> 1);
          if (d == 0 || same_cell(hi, lo, h, l, mid, d)) in = mid;
          else out = mid;
        }
        end = in + 1;
      }
      const int32_t parent = d == before + 1 ? up : (int32_t)(id - 1);
      by_depth[start[d] + atomicAdd(&here[d], 1u)] = id;
      o_parent[id] = parent;
      o_depth[id] = (uint8_t)d;
      o_first[id] = (uint32_t)i;
      o_last[id] = (uint32_t)(end - 1);
      if (parent >= 0) slots[(int64_t)parent * 8 + digit_at(h, l, d)] = id;
    }
    const int ld = (c ? after : before) + 1;
    const int32_t lp = c ? (int32_t)(id0 + c - 1) : up;
    leaf_depth[i] = (uint8_t)ld;
    if (lp >= 0 && ld <= KEY_LEVELS) slots[(int64_t)lp * 8 + digit_at(h, l, ld)] = (uint32_t)i | LEAF_BIT;
    if (c) deep = (uint32_t)(after + 1);
  }
  // deepest leaf bound: one atomic per warp (one per thread on a single
  // address serialised the kernel)
  deep = __reduce_max_sync(0xffffffffu, deep);
  if ((threadIdx.x & 31) == 0 && deep) atomicMax(max_depth, deep);
}

// ---------------------------------------------------------------------------
// bottom-up aggregation (octree.rs:547-629), float64, reference order
// ---------------------------------------------------------------------------
// Mass and centre of mass of an octree child (leaf: the particle).
__device__ __forceinline__ void child_moments(uint32_t c, double scale, const uint32_t* __restrict__ qx,
                                              const uint32_t* __restrict__ qy, const uint32_t* __restrict__ qz,
                                              const double* __restrict__ pmass, const double* o_mass,
                                              const double* o_com, double* m, double* x, double* y, double* z) {
  if (c & LEAF_BIT) {
    const uint32_t j = c & ~LEAF_BIT;
    *m = pmass[j];
    *x = decode(qx[j], scale);
    *y = decode(qy[j], scale);
    *z = decode(qz[j], scale);
  } else {
    *m = __ldcg(&o_mass[c]);
    *x = __ldcg(&o_com[3 * (int64_t)c]);
    *y = __ldcg(&o_com[3 * (int64_t)c + 1]);
    *z = __ldcg(&o_com[3 * (int64_t)c + 2]);
  }
}

// Moments of the internal nodes at one depth (octree.rs:547-629) from their
// children, which are leaves or nodes one level deeper (finished by the
// previous launch): mass and centre of mass summed over the children in
// octant order, then the quadrupole by the parallel-axis theorem
// (outer_traceless :197-207), all float64 in the reference's operation order.
// QUAD: also the quadrupole tensors (the walk reads mass and centre of mass
// only; the quadrupoles are made when the tree is exported).
// Returns the number of children.
template <bool QUAD>
__device__ __forceinline__ uint32_t aggregate_node(uint32_t P, double scale, const uint32_t* __restrict__ qx,
                                               const uint32_t* __restrict__ qy, const uint32_t* __restrict__ qz,
                                               const double* __restrict__ pmass, const uint32_t* __restrict__ slots,
                                               double* o_mass, double* o_com, double* o_quad, double inv_scale,
                                               uint4* __restrict__ walk, uint8_t* __restrict__ kids) {
  // pass 1: mass and centre of mass over the children in octant order
  uint32_t cs[8], nk = 0;  // children, internal ones in the high half byte
  double mt = 0.0, ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const uint32_t c = slots[(int64_t)P * 8 + s];
    cs[s] = c;
    if (c == EMPTY_SLOT) continue;
    nk += (c & LEAF_BIT) ? 1u : 17u;
    double m, x, y, z;
    child_moments(c, scale, qx, qy, qz, pmass, o_mass, o_com, &m, &x, &y, &z);
    mt = dadd(mt, m);
    ax = dadd(ax, dmul(x, m));
    ay = dadd(ay, dmul(y, m));
    az = dadd(az, dmul(z, m));
  }
  double comx = 0.0, comy = 0.0, comz = 0.0;
  if (mt > 0.0) {
    comx = ddiv(ax, mt);
    comy = ddiv(ay, mt);
    comz = ddiv(az, mt);
  }
  kids[P] = (uint8_t)nk;
  {  // the walk's fixed-point centre of mass (in [0, 2^32]) and float mass
    const double v[3] = {comx, comy, comz};
    uint32_t q[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) q[d] = (uint32_t)((unsigned long long)llrint(v[d] * inv_scale) & 0xFFFFFFFFull);
    walk[P] = make_uint4(q[0], q[1], q[2], __float_as_uint((float)mt));
  }
  if (!QUAD) {
    __stcg(&o_mass[P], mt);
    __stcg(&o_com[3 * (int64_t)P], comx);
    __stcg(&o_com[3 * (int64_t)P + 1], comy);
    __stcg(&o_com[3 * (int64_t)P + 2], comz);
    return nk & 15u;
  }
  // pass 2: the children are read again (cache hits) rather than held in registers
  double qd[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int s = 0; s < 8; ++s) {
    const uint32_t c = cs[s];
    if (c == EMPTY_SLOT) continue;
    double m, x, y, z;
    child_moments(c, scale, qx, qy, qz, pmass, o_mass, o_com, &m, &x, &y, &z);
    if (m == 0.0) continue;
    const double sx = dsub(x, comx), sy = dsub(y, comy), sz = dsub(z, comz);
    const double s2 = dadd(dadd(dmul(sx, sx), dmul(sy, sy)), dmul(sz, sz));
    const double m3 = dmul(m, 3.0);
    double oq[6];
    oq[0] = dmul(m, dsub(dmul(dmul(3.0, sx), sx), s2));
    oq[1] = dmul(dmul(m3, sx), sy);
    oq[2] = dmul(dmul(m3, sx), sz);
    oq[3] = dmul(m, dsub(dmul(dmul(3.0, sy), sy), s2));
    oq[4] = dmul(dmul(m3, sy), sz);
    oq[5] = dmul(m, dsub(dmul(dmul(3.0, sz), sz), s2));
    if (c & LEAF_BIT) {
#pragma unroll
      for (int k = 0; k < 6; ++k) qd[k] = dadd(qd[k], dadd(0.0, oq[k]));
    } else {
#pragma unroll
      for (int k = 0; k < 6; ++k) qd[k] = dadd(qd[k], dadd(__ldcg(&o_quad[6 * (int64_t)c + k]), oq[k]));
    }
  }
  __stcg(&o_mass[P], mt);
  __stcg(&o_com[3 * (int64_t)P], comx);
  __stcg(&o_com[3 * (int64_t)P + 1], comy);
  __stcg(&o_com[3 * (int64_t)P + 2], comz);
#pragma unroll
  for (int k = 0; k < 6; ++k) __stcg(&o_quad[6 * (int64_t)P + k], qd[k]);
  return nk & 15u;
}

// Space for the walk records of this lane's node (nk children, 0: none), one
// atomic per warp: the ranges need no order among the nodes, so no prefix sum.
// All lanes of the warp call it.
__device__ __forceinline__ void reserve_children(bool live, uint32_t P, uint32_t nk, uint32_t* total,
                                                 uint32_t* __restrict__ child_first) {
  const int lane = threadIdx.x & 31;
  if (!live) nk = 0u;
  uint32_t x = nk;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  uint32_t base = 0;
  if (lane == 31 && x) base = atomicAdd(total, x);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (live) child_first[P] = base + x - nk;
}

template <bool QUAD>
__global__ void k_aggregate_level(const uint32_t* __restrict__ nodes, int64_t count, double scale,
                                  const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                                  const uint32_t* __restrict__ qz, const double* __restrict__ pmass,
                                  const uint32_t* __restrict__ slots, double* o_mass, double* o_com, double* o_quad,
                                  double inv_scale, uint4* __restrict__ walk, uint8_t* __restrict__ kids,
                                  uint32_t* total, uint32_t* __restrict__ child_first) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool live = i < count;
  const uint32_t P = live ? nodes[i] : 0u;
  uint32_t nk = 0u;
  if (live) nk = aggregate_node<QUAD>(P, scale, qx, qy, qz, pmass, slots, o_mass, o_com, o_quad, inv_scale, walk, kids);
  if (total) reserve_children(live, P, nk, total, child_first);
}

// Small trees in one block: every level from the deepest up with a block
// barrier between levels, in place of one launch per depth.
constexpr int AGG_SMALL_THREADS = 512;
template <bool QUAD>
__global__ void __launch_bounds__(AGG_SMALL_THREADS)
    k_aggregate_small(const uint32_t* __restrict__ off, const uint32_t* __restrict__ by_depth, double scale,
                      const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy, const uint32_t* __restrict__ qz,
                      const double* __restrict__ pmass, const uint32_t* __restrict__ slots, double* o_mass,
                      double* o_com, double* o_quad, double inv_scale, uint4* __restrict__ walk,
                      uint8_t* __restrict__ kids, uint32_t* total, uint32_t* __restrict__ child_first) {
  for (int d = DEPTH_BINS - 1; d >= 0; --d) {
    if (off[d] == off[d + 1]) continue;  // the same for the whole block
    const uint32_t end = off[d + 1];
    for (uint32_t i0 = off[d]; i0 < end; i0 += AGG_SMALL_THREADS) {
      const uint32_t i = i0 + threadIdx.x;
      const bool live = i < end;
      const uint32_t P = live ? by_depth[i] : 0u;
      uint32_t nk = 0u;
      if (live)
        nk = aggregate_node<QUAD>(P, scale, qx, qy, qz, pmass, slots, o_mass, o_com, o_quad, inv_scale, walk, kids);
      if (total) reserve_children(live, P, nk, total, child_first);
    }
    __syncthreads();
  }
}

// Up to here one block is faster than the launches per level.
constexpr int64_t AGG_SMALL_MAX = 8192;

// Cell centre and |Q|_F of each internal node (relative opening criterion).
// The node's octant path is the first `depth` digits of any of its particles'
// keys (sorted order: o_first); the centre follows child_center level by
// level in float64 as k_tree_keys does.
__global__ void k_cell_q(int64_t n_int, double inv_scale, const TreeParams* __restrict__ prm,
                         const uint8_t* __restrict__ o_depth, const uint32_t* __restrict__ o_first,
                         const uint64_t* __restrict__ key_hi, const uint64_t* __restrict__ key_lo,
                         const double* __restrict__ o_quad, uint4* __restrict__ out) {
  int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (id >= n_int) return;
  const int dep = o_depth[id];
  const uint32_t p = o_first[id];
  double c[3] = {prm->center[0], prm->center[1], prm->center[2]};
  double h = prm->half;
  for (int l = 1; l <= dep && l <= KEY_LEVELS; ++l) {
    const uint64_t w = l <= KEY_LEVELS / 2 ? key_hi[p] : key_lo[p];
    const int ll = l <= KEY_LEVELS / 2 ? l : l - KEY_LEVELS / 2;
    const uint32_t digit = (uint32_t)(w >> (63 - 3 * ll)) & 7u;
    const double q = dmul(h, 0.5);
#pragma unroll
    for (int d = 0; d < 3; ++d) c[d] = dadd(c[d], ((digit >> d) & 1u) ? q : -q);
    h = q;
  }
  uint32_t cq[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double u = c[d] * inv_scale;  // fixed point, wrapped like positions
    cq[d] = (uint32_t)((unsigned long long)llrint(u) & 0xFFFFFFFFull);
  }
  const double* Q = o_quad + 6 * id;
  double f2 = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) f2 = fma(Q[k], Q[k], f2);
  out[id] = make_uint4(cq[0], cq[1], cq[2], __float_as_uint((float)sqrt(f2)));
}

// ---------------------------------------------------------------------------
// walk records: children of each internal node contiguous
// ---------------------------------------------------------------------------
// One thread per node gathers its children's records, internal ones first, into
// the node's range (1 + child_first[P] onward; the root's own record is number 0).
__global__ void k_walk_records(int64_t n_int, const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                               const uint32_t* __restrict__ qz, const float* __restrict__ massf,
                               const uint8_t* __restrict__ leaf_depth, const uint4* __restrict__ walk,
                               const uint8_t* __restrict__ o_depth, const uint8_t* __restrict__ kids,
                               const uint32_t* __restrict__ child_first, const uint32_t* __restrict__ slots,
                               WalkNode* __restrict__ recs) {
  const int64_t P = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (P >= n_int) return;
  auto internal = [&](uint32_t c) {
    const uint4 w = walk[c];
    const uint32_t k = kids[c];
    WalkNode r;
    r.cq[0] = w.x;
    r.cq[1] = w.y;
    r.cq[2] = w.z;
    r.mass = __uint_as_float(w.w);
    r.first = 1u + child_first[c];
    r.info = (k & 15u) | ((uint32_t)o_depth[c] << 4) | ((k >> 4) << 12);
    r.ref = c;
    r.pad = 0;
    return r;
  };
  if (P == 0) recs[0] = internal(0u);
  WalkNode* out = recs + 1 + (int64_t)child_first[P];
  uint32_t cs[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    cs[s] = slots[P * 8 + s];
    if (!(cs[s] & LEAF_BIT)) *out++ = internal(cs[s]);  // (EMPTY_SLOT has the leaf bit)
  }
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    if (!(cs[s] & LEAF_BIT) || cs[s] == EMPTY_SLOT) continue;
    const uint32_t j = cs[s] & ~LEAF_BIT;
    WalkNode r;
    r.cq[0] = qx[j];
    r.cq[1] = qy[j];
    r.cq[2] = qz[j];
    r.mass = massf[j];
    r.first = 0;
    r.info = ((uint32_t)leaf_depth[j] << 4) | WN_LEAF;
    r.ref = j;
    r.pad = 0;
    *out++ = r;
  }
}

// ---------------------------------------------------------------------------
// walk groups: maximal subtrees of <= group_max particles, consecutive small
// siblings packed together; cells above pack_depth are always split, and
// their children never packed, so no group is wider than a cell of that depth
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t child_count(uint32_t c, const uint32_t* __restrict__ o_first,
                                                const uint32_t* __restrict__ o_last) {
  return (c & LEAF_BIT) ? 1u : o_last[c] - o_first[c] + 1u;
}
__device__ __forceinline__ uint32_t child_first_particle(uint32_t c, const uint32_t* __restrict__ o_first) {
  return (c & LEAF_BIT) ? (c & ~LEAF_BIT) : o_first[c];
}

// Two looks at the children of a node, the first to count its groups.  RESERVE:
// a warp takes the slots of its nodes' groups at once, so the groups come nearly
// in the order of the nodes.  COUNT and WRITE: the slots are a prefix sum in node
// order, made between two launches; neighbouring groups then walk at the same
// time, which is worth more in large boxes (walk of 256^3 40.7 -> 40.5 ms, accurate
// 128^3 7.55 -> 7.47) than the four launches it costs (12 us).
constexpr int64_t GROUPS_RESERVE_MAX = 262144;
enum { GROUPS_RESERVE = 0, GROUPS_COUNT = 1, GROUPS_WRITE = 2 };
template <int MODE>
__global__ void k_groups(int64_t n_int, int group_max, int pack_depth, const uint8_t* __restrict__ o_depth,
                         const uint32_t* __restrict__ slots, const uint32_t* __restrict__ o_first,
                         const uint32_t* __restrict__ o_last, uint32_t* __restrict__ count,
                         uint32_t* __restrict__ per_node, uint32_t* __restrict__ gfirst,
                         uint32_t* __restrict__ gsize) {
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool live = id < n_int;
  const uint32_t mine = live ? o_last[id] - o_first[id] + 1u : 0u;
  const int dep = live ? o_depth[id] : 0;
  const bool split = live && (mine > (uint32_t)group_max || dep < pack_depth);
  const bool whole = live && !split && id == 0;  // the whole tree fits in one group
  uint32_t w = MODE == GROUPS_WRITE && live ? per_node[id] : 0u;
  for (int pass = MODE == GROUPS_WRITE ? 1 : 0; pass < 2; ++pass) {
    uint32_t ng = 0;
    auto emit = [&](uint32_t first, uint32_t n) {
      if (pass) {
        gfirst[w + ng] = first;
        gsize[w + ng] = n;
      }
      ++ng;
    };
    if (split) {
      const uint32_t pack_max = dep < pack_depth ? 0u : (uint32_t)group_max;
      uint32_t run_first = 0, run_n = 0;
      for (int s = 0; s < 8; ++s) {
        const uint32_t c = slots[id * 8 + s];
        if (c == EMPTY_SLOT) continue;
        const uint32_t k = child_count(c, o_first, o_last);
        const bool apart = k > (uint32_t)group_max || (k > 1u && dep + 1 < pack_depth);
        if (run_n && (apart || run_n + k > pack_max)) {
          emit(run_first, run_n);
          run_n = 0;
        }
        if (apart) continue;
        if (!run_n) run_first = child_first_particle(c, o_first);
        run_n += k;
      }
      if (run_n) emit(run_first, run_n);
    } else if (whole) {
      emit(o_first[0], mine);
    }
    if (MODE == GROUPS_COUNT) {
      if (live) per_node[id] = ng;
      return;
    }
    if (pass == 0) {
      const int lane = threadIdx.x & 31;
      uint32_t x = ng;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      uint32_t base = 0;
      if (lane == 31 && x) base = atomicAdd(count, x);
      w = __shfl_sync(0xffffffffu, base, 31) + x - ng;
      if (!__any_sync(0xffffffffu, ng != 0u)) return;
    }
  }
}

// ---------------------------------------------------------------------------
// Hilbert keys (crates/gadget-ng-parallel/src/sfc.rs:95-204)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t coords_to_hilbert(uint32_t ix, uint32_t iy, uint32_t iz, uint32_t p) {
  uint32_t x[3] = {ix, iy, iz};
  const uint32_t m = 1u << (p - 1);
  for (uint32_t q = m; q > 1; q >>= 1) {
    const uint32_t pm = q - 1;
#pragma unroll
    for (int i = 2; i >= 0; --i) {
      if (x[i] & q) {
        x[0] ^= pm;
      } else {
        uint32_t t = (x[0] ^ x[i]) & pm;
        x[0] ^= t;
        x[i] ^= t;
      }
    }
  }
  x[1] ^= x[0];
  x[2] ^= x[1];
  uint32_t t = 0;
  for (uint32_t q = m; q > 1; q >>= 1)
    if (x[2] & q) t ^= q - 1;
  x[0] ^= t;
  x[1] ^= t;
  x[2] ^= t;
  uint64_t h = 0;
  for (uint32_t k = 0; k < p; ++k) {
    h = (h << 1) | ((x[0] >> k) & 1u);
    h = (h << 1) | ((x[1] >> k) & 1u);
    h = (h << 1) | ((x[2] >> k) & 1u);
  }
  return h;
}

__device__ __forceinline__ uint32_t hilbert_coord(double x, double lo, double len) {
  double v = ddiv(dsub(x, lo), len);
  v = v < 0.0 ? 0.0 : (v > 1.0 - F64_EPSILON ? 1.0 - F64_EPSILON : v);  // f64::clamp
  return (uint32_t)dmul(v, 2097152.0);
}

__global__ void k_hilbert(const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                          const uint32_t* __restrict__ qz, const uint32_t* __restrict__ id, int64_t n, double scale,
                          const TreeParams* __restrict__ prm, uint64_t* __restrict__ keys,
                          uint32_t* __restrict__ vals) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t ix = hilbert_coord(decode(qx[i], scale), prm->hlo[0], prm->hlen[0]);
  const uint32_t iy = hilbert_coord(decode(qy[i], scale), prm->hlo[1], prm->hlen[1]);
  const uint32_t iz = hilbert_coord(decode(qz[i], scale), prm->hlo[2], prm->hlen[2]);
  keys[i] = coords_to_hilbert(ix, iy, iz, 21);
  vals[i] = id ? id[i] : (uint32_t)i;
}

// spread_bits (crates/gadget-ng-parallel/src/sfc.rs:39-47): the 21 low bits of
// x to every third bit position.
__device__ __forceinline__ uint64_t spread3(uint64_t x) {
  x &= 0x1FFFFFull;
  x = (x | (x << 32)) & 0x1F00000000FFFFull;
  x = (x | (x << 16)) & 0x1F0000FF0000FFull;
  x = (x | (x << 8)) & 0x100F00F00F00F00Full;
  x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

// particle_morton (sfc.rs:54-81): the coordinates normalised and quantised as
// for the Hilbert keys, interleaved x | y << 1 | z << 2.
__global__ void k_morton(const uint32_t* __restrict__ qx, const uint32_t* __restrict__ qy,
                         const uint32_t* __restrict__ qz, const uint32_t* __restrict__ id, int64_t n, double scale,
                         const TreeParams* __restrict__ prm, uint64_t* __restrict__ keys,
                         uint32_t* __restrict__ vals) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t ix = hilbert_coord(decode(qx[i], scale), prm->hlo[0], prm->hlen[0]);
  const uint32_t iy = hilbert_coord(decode(qy[i], scale), prm->hlo[1], prm->hlen[1]);
  const uint32_t iz = hilbert_coord(decode(qz[i], scale), prm->hlo[2], prm->hlen[2]);
  keys[i] = spread3(ix) | (spread3(iy) << 1) | (spread3(iz) << 2);
  vals[i] = id ? id[i] : (uint32_t)i;
}

__device__ __forceinline__ void mask_path(uint64_t hi, uint64_t lo, int depth, uint64_t* oh, uint64_t* ol) {
  if (depth <= 0) { *oh = 0; *ol = 0; return; }
  if (depth <= 21) {
    int keep = 3 * depth;  // bits 62..63-keep
    uint64_t m = keep >= 63 ? 0x7FFFFFFFFFFFFFFFull : (((1ull << keep) - 1) << (63 - keep));
    *oh = hi & m;
    *ol = 0;
  } else {
    int keep = 3 * (depth - 21);
    uint64_t m = keep >= 63 ? 0x7FFFFFFFFFFFFFFFull : (((1ull << keep) - 1) << (63 - keep));
    *oh = hi;
    *ol = lo & m;
  }
}

__global__ void k_export_paths(int64_t n, int64_t n_int, const uint8_t* __restrict__ o_depth,
                               const uint32_t* __restrict__ o_first, const uint8_t* __restrict__ leaf_depth,
                               const uint64_t* __restrict__ hi, const uint64_t* __restrict__ lo, uint64_t* nh,
                               uint64_t* nl, uint64_t* lh, uint64_t* ll) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n_int) {
    uint32_t f = o_first[i];
    mask_path(hi[f], lo[f], o_depth[i], &nh[i], &nl[i]);
  }
  if (i < n) mask_path(hi[i], lo[i], leaf_depth ? leaf_depth[i] : 0, &lh[i], &ll[i]);
}

}  // namespace

// ===========================================================================
// launchers
// ===========================================================================
void launch_bbox_root(const Particles& p, int64_t n, double box, TreeBuffers& t, cudaStream_t s) {
  k_bbox_init<<<1, 32, 0, s>>>(t.bbox);
  TPM_LAUNCH_CHECK();
  k_bbox<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(p.qx, p.qy, p.qz, n, t.bbox);
  TPM_LAUNCH_CHECK();
  k_root<<<1, 32, 0, s>>>(t.bbox, box / TWO32, t.params);
  TPM_LAUNCH_CHECK();
}

void launch_tree_keys(const Particles& p, int64_t n, double box, TreeBuffers& t, cudaStream_t s) {
  k_tree_keys<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(p.qx, p.qy, p.qz, n, box / TWO32, t.params, t.key_hi,
                                                          t.perm);
  TPM_LAUNCH_CHECK();
}

void launch_fix_ties(const Particles& p, int64_t n, double box, TreeBuffers& t, cudaStream_t s) {
  k_tie_low<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(p.qx, p.qy, p.qz, n, box / TWO32, t.params, t.key_hi,
                                                        t.perm, t.key_lo_tmp);
  TPM_LAUNCH_CHECK();
  k_fix_ties<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(n, t.key_hi, t.perm, t.key_lo_tmp, t.key_lo, t.err);
  TPM_LAUNCH_CHECK();
}

void launch_permute(const Particles& src, const Particles& dst, int64_t n, const uint32_t* perm, cudaStream_t s) {
  k_permute<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(src, dst, n, perm);
  TPM_LAUNCH_CHECK();
}

void launch_levels(int64_t n, TreeBuffers& t, cudaStream_t s) {
  if (n < 2) return;
  TPM_CUDA(cudaMemsetAsync(t.depth_tab, 0, DEPTH_BINS * sizeof(uint32_t), s));
  k_levels<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(n, t.key_hi, t.key_lo, t.lev, t.oct_count, t.depth_tab);
  TPM_LAUNCH_CHECK();
  k_depth_offsets<<<1, 32, 0, s>>>(t.depth_tab);
  TPM_LAUNCH_CHECK();
}

void launch_octree_nodes(int64_t n, int64_t n_int, TreeBuffers& t, cudaStream_t s) {
  TPM_CUDA(cudaMemsetAsync(t.o_slots, 0xFF, (size_t)n_int * 8 * sizeof(uint32_t), s));
  k_oct_nodes<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(n, n_int, t.lev, t.key_hi, t.key_lo, t.oct_base, t.o_parent,
                                                          t.o_depth, t.o_first, t.o_last, t.leaf_depth, t.o_slots,
                                                          &t.scalars[2], t.depth_tab + 2 * DEPTH_BINS + 1, t.o_cnt);
  TPM_LAUNCH_CHECK();
}

// Level by level from the deepest internal nodes to the root: each launch
// finishes one depth, so every node reads finished children without atomics
// or fences.
void launch_aggregate(const Particles& p, int64_t n, int64_t n_int, double box, TreeBuffers& t, const uint32_t* counts,
                      cudaStream_t s, bool with_quad, bool records) {
  (void)n;
  if (n_int <= 0) return;
  const double scale = box / TWO32, inv_scale = TWO32 / box;
  uint32_t* total = records ? &t.scalars[3] : nullptr;  // zero since the node count was made
  if (n_int <= AGG_SMALL_MAX) {
    auto k = with_quad ? k_aggregate_small<true> : k_aggregate_small<false>;
    k<<<1, AGG_SMALL_THREADS, 0, s>>>(t.depth_tab + DEPTH_BINS, t.o_cnt, scale, p.qx, p.qy, p.qz, p.mass, t.o_slots,
                                      t.o_mass, t.o_com, t.o_quad, inv_scale, t.o_walk, t.o_kids, total,
                                      t.o_child_first);
    TPM_LAUNCH_CHECK();
    return;
  }
  int64_t offset[DEPTH_BINS + 1];
  offset[0] = 0;
  for (int d = 0; d < DEPTH_BINS; ++d) offset[d + 1] = offset[d] + counts[d];
  if (offset[DEPTH_BINS] != n_int) throw Error(2, "octree depth buckets do not add up to the node count");
  auto k = with_quad ? k_aggregate_level<true> : k_aggregate_level<false>;
  for (int d = DEPTH_BINS - 1; d >= 0; --d) {
    if (counts[d] == 0) continue;
    k<<<grid_for(counts[d], 128, 1ll << 30), 128, 0, s>>>(t.o_cnt + offset[d], counts[d], scale, p.qx, p.qy, p.qz,
                                                          p.mass, t.o_slots, t.o_mass, t.o_com, t.o_quad, inv_scale,
                                                          t.o_walk, t.o_kids, total, t.o_child_first);
    TPM_LAUNCH_CHECK();
  }
}

void launch_cell_q(int64_t n_int, double box, TreeBuffers& t, cudaStream_t s) {
  if (n_int <= 0) return;
  k_cell_q<<<grid_for(n_int, 256, 1ll << 30), 256, 0, s>>>(n_int, TWO32 / box, t.params, t.o_depth, t.o_first,
                                                           t.key_hi, t.key_lo, t.o_quad, t.o_cell);
  TPM_LAUNCH_CHECK();
}

void launch_walk_records(const Particles& p, int64_t n_int, TreeBuffers& t, cudaStream_t s) {
  k_walk_records<<<grid_for(n_int, 128, 1ll << 30), 128, 0, s>>>(n_int, p.qx, p.qy, p.qz, p.massf, t.leaf_depth,
                                                                 t.o_walk, t.o_depth, t.o_kids, t.o_child_first,
                                                                 t.o_slots, t.recs);
  TPM_LAUNCH_CHECK();
}

void launch_groups(int64_t n_int, int group_max, int pack_depth, TreeBuffers& t, void* scan_scratch, cudaStream_t s) {
  const unsigned grid = grid_for(n_int, 256, 1ll << 30);
  auto run = [&](auto k) {
    k<<<grid, 256, 0, s>>>(n_int, group_max, pack_depth, t.o_depth, t.o_slots, t.o_first, t.o_last, &t.scalars[1],
                           t.grp_base, t.grp_first, t.grp_size);
    TPM_LAUNCH_CHECK();
  };
  // (the sum's scratch covers four entries per particle: a tree of chains, with
  // more nodes than that, reserves too)
  if (n_int <= GROUPS_RESERVE_MAX || n_int > 4 * (t.cap_groups - 1)) {
    run(k_groups<GROUPS_RESERVE>);
    return;
  }
  run(k_groups<GROUPS_COUNT>);
  exclusive_scan_u32(t.grp_base, t.grp_base, n_int, &t.scalars[1], scan_scratch, s);
  run(k_groups<GROUPS_WRITE>);
}

void launch_hilbert_keys(const Particles& p, int64_t n, double box, const TreeParams* prm, uint64_t* keys,
                         uint32_t* vals, cudaStream_t s) {
  k_hilbert<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(p.qx, p.qy, p.qz, p.id, n, box / TWO32, prm, keys, vals);
  TPM_LAUNCH_CHECK();
}

void launch_morton_keys(const Particles& p, int64_t n, double box, const TreeParams* prm, uint64_t* keys,
                        uint32_t* vals, cudaStream_t s) {
  k_morton<<<grid_for(n, 256, 1ll << 30), 256, 0, s>>>(p.qx, p.qy, p.qz, p.id, n, box / TWO32, prm, keys, vals);
  TPM_LAUNCH_CHECK();
}

void launch_export_paths(int64_t n, int64_t n_int, const TreeBuffers& t, uint64_t* node_hi, uint64_t* node_lo,
                         uint64_t* leaf_hi, uint64_t* leaf_lo, cudaStream_t s) {
  int64_t m = n > n_int ? n : n_int;
  k_export_paths<<<grid_for(m, 256, 1ll << 30), 256, 0, s>>>(n, n_int, t.o_depth, t.o_first,
                                                             n > 1 ? t.leaf_depth : nullptr, t.key_hi, t.key_lo,
                                                             node_hi, node_lo, leaf_hi, leaf_lo);
  TPM_LAUNCH_CHECK();
}

}  // namespace tpm
