// Short-range TreePM walk, one warp per target group.
//
// Semantics (crates/gadget-ng-treepm/src/short_range.rs:274-333, periodic;
// :157-208, aperiodic): for each target particle the reference pops nodes
// from a stack, drops a node whose AABB (centred on its centre of mass, half
// side = the cell's half side) lies beyond r_cut, adds the pair force of a
// leaf (periodic walk: only if the bare minimum-image distance is within
// r_cut), takes an internal node whose half side is below 0.1 r_cut as a
// monopole (unless its centre of mass sits on the target), and otherwise
// opens it.  An internal node's cull hides all its descendants, so whether a
// target interacts with a node depends on every ancestor on its path.
//
// Warp design: the 32 lanes hold up to 32 target particles from one compact
// subtree.  The warp walks the tree once for all of them: each range of nodes
// on its stack carries a 32-bit mask of the targets that still see it.  Nodes
// are classified against the group's bounding box in FP32 with a safety margin
// (certainly culled / certainly kept for every target / undecided); undecided
// internal nodes get a per-target test before they are pushed, which refines
// the mask, so the hierarchical culls of the reference are reproduced exactly.
// Terminal nodes (leaves and monopole-depth cells) go to interaction lists in
// shared memory; the lanes evaluate a list against the group's targets with
// each target's own final test fused into the pair kernel (a group of c
// targets gives every target 32 / c lanes, each on a share of the entries).
// The running per-target sums, the targets' positions and the group box stay
// in shared memory.  Any decision that falls inside a narrow band around r_cut
// is re-evaluated in float64 with the reference's exact expression, so the
// interaction set equals the reference's.  Pair arithmetic is FP32: exact
// fixed-point differences rounded once, rsqrt / ex2 hardware approximations, the
// A&S 7.1.26 erfc as a polynomial where that holds out to the farthest pair,
// Kahan-compensated per-target sums.
//
// What bounds it (lattice of 128^3, 84 k groups, B200 at 1965 MHz): issue slots.
// 11.28e9 warp instructions took 11.3 ms at 88 % issue before the pair loop
// took two entries per iteration in f32x2 arithmetic (63 instructions for
// two entries, ~106 before) and the traversal was split into open and item
// steps; 5.74e9 take 6.93 ms at 73 % now (62.7 -> 39.3 ms on the clustered
// 256^3 box).  Two thirds are the pair loop (60 per iteration), its FMA pipe
// 56 % busy.  The accurate mode took the same steps later: 10.3 -> 7.4 ms on the
// clustered 128^3 box against its former traversal (32 children of a popped
// batch per step, opening tests at pop time).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "tree.cuh"
#include "walk.cuh"

namespace tpm {
namespace {

constexpr int WALK_WARPS = 4;
constexpr int WALK_THREADS = WALK_WARPS * 32;
// List capacities (leaves, monopoles).  Longer lists are flushed less often (30
// times per group at 64 entries, each time a start of both pair loops and a
// compensated add), but leave less L1 cache to the tree.  Parity, clustered
// 256^3 / 128^3 / clustered 99^3, walk ms: 64 entries 40.6 / 7.17 / 4.05, 96 39.7 /
// 7.02 / 3.97, 128 39.3 / 6.93 / 3.95, 192 leaves and 64 monopoles 39.1 / 6.93 /
// 4.07, 256 and 64 39.2 / 6.92 / 4.07.  Accurate 128^3: 64 7.46, 96 7.53, 128 7.79.
template <bool ACC> constexpr int chunk_l() { return ACC ? 64 : 128; }
template <bool ACC> constexpr int chunk_m() { return ACC ? 64 : 128; }


// An interaction list in shared memory, kept in pairs of entries so that the
// pair loop reads both entries of a packed (f32x2) operand with one load:
// source positions relative to the middle of the group's box in walk units (the
// exact difference of the coordinates, rounded once: the float64 band settles
// every borderline cut, and CLOSE walks take the exact difference of the target
// and the source where the two are near), masses, the masks of targets that see
// them, the nodes
// (LEAF_BIT | particle for leaves) and, where a list needs them, cull half
// sides.
template <bool HALF> struct __align__(16) EntryPair {
  float4 xy;   // x0 x1 y0 y1
  float4 zm;   // z0 z1 m0 m1
  uint2 mask;
  uint2 node;
};
template <> struct __align__(16) EntryPair<true> {
  float4 xy;
  float4 zm;
  uint2 mask;
  uint2 node;
  float2 h;
};
template <int CAP, bool HALF> struct List {
  static_assert(CAP % 2 == 0, "entries are evaluated two at a time");
  EntryPair<HALF> pair[CAP / 2];
  // word w of entry e: members of a pair interleave its two entries
  __device__ __forceinline__ static float* word(EntryPair<HALF>* pair, int e) {
    return reinterpret_cast<float*>(&pair[e >> 1]) + (e & 1);
  }
  __device__ __forceinline__ float* word(int e) { return word(pair, e); }
  __device__ __forceinline__ const float* word(int e) const {
    return reinterpret_cast<const float*>(&pair[e >> 1]) + (e & 1);
  }
  __device__ __forceinline__ void put(int e, float x, float y, float z, float m, float half, uint32_t see, uint32_t nd) {
    put(pair, e, x, y, z, m, half, see, nd);
  }
  __device__ __forceinline__ static void put(EntryPair<HALF>* pair, int e, float x, float y, float z, float m, float half,
                                             uint32_t see, uint32_t nd) {
    float* w = word(pair, e);
    w[0] = x;
    w[2] = y;
    w[4] = z;
    w[6] = m;
    w[8] = __uint_as_float(see);
    w[10] = __uint_as_float(nd);
    if (HALF) w[12] = half;
  }
  // nobody sees the second half of an odd list's last pair
  __device__ __forceinline__ void close(int n) {
    if (n & 1) word(n)[8] = 0.f;
  }
};

// Packed pairs of floats (PTX f32x2, one instruction for both halves).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// min(|a|, |b|, |c|) in one instruction
__device__ __forceinline__ float min3_abs(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// a - b in quanta: the minimum image (modulo 2^32), or in the aperiodic walk the
// difference itself, up to a whole box.
__device__ __forceinline__ float rel(uint32_t a, uint32_t b, int periodic) {
  if (periodic) return (float)(int32_t)(a - b);
  return a >= b ? (float)(a - b) : -(float)(b - a);
}


// h0 * 2^-dep by exponent arithmetic: h0 (the root half side in walk units,
// O(r_cut / cell)) stays a normal float for every tree depth (-1 <= dep < 64).
__device__ __forceinline__ float half_side(float h0, int dep) {
  return __int_as_float(__float_as_int(h0) - dep * (1 << 23));
}

// ---- float64 decisions with the reference's expressions -------------------
__device__ __forceinline__ double aabb_axis(double dc, double h) {
  double e = dsub(fabs(dc), h);
  return e > 0.0 ? e : 0.0;
}

// min_dist2_to_aabb_periodic (short_range.rs:72-84) or its aperiodic twin (:173-181).
__device__ __forceinline__ double d2_aabb(const double xi[3], const double com[3], double h, double box, int periodic) {
  double e[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double dc = dsub(com[a], xi[a]);
    if (periodic) dc = minimum_image(dc, box);
    e[a] = aabb_axis(dc, h);
  }
  return dadd(dadd(dmul(e[0], e[0]), dmul(e[1], e[1])), dmul(e[2], e[2]));
}

__device__ __forceinline__ void target_pos(const WalkArgs& a, uint32_t p, double xi[3]) {
  xi[0] = decode(a.qx[p], a.scale);
  xi[1] = decode(a.qy[p], a.scale);
  xi[2] = decode(a.qz[p], a.scale);
}

__device__ __forceinline__ void node_com(const WalkArgs& a, uint32_t node, double c[3]) {
  if (node & LEAF_BIT) {
    uint32_t j = node & ~LEAF_BIT;
    c[0] = decode(a.qx[j], a.scale);
    c[1] = decode(a.qy[j], a.scale);
    c[2] = decode(a.qz[j], a.scale);
  } else {
    c[0] = a.o_com[3 * (int64_t)node];
    c[1] = a.o_com[3 * (int64_t)node + 1];
    c[2] = a.o_com[3 * (int64_t)node + 2];
  }
}

// Does target p keep open internal node `node` (cull test only)?
__device__ __forceinline__ bool exact_open_pass(const WalkArgs& a, uint32_t p, uint32_t node) {
  double xi[3], c[3];
  target_pos(a, p, xi);
  node_com(a, node, c);
  double h = ldexp(a.h0, -(int)a.depth[node]);
  return !(d2_aabb(xi, c, h, a.box, a.periodic) > a.rc2);
}

// Terminal node decision: 0 = skip, 1 = interact, 2 = open for this target
// (monopole whose centre of mass coincides with the target).
__device__ __forceinline__ int exact_terminal(const WalkArgs& a, uint32_t p, uint32_t node) {
  double xi[3], c[3];
  target_pos(a, p, xi);
  node_com(a, node, c);
  if (node & LEAF_BIT) {
    uint32_t j = node & ~LEAF_BIT;
    if (a.periodic) {
      double r[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) r[k] = minimum_image(dsub(c[k], xi[k]), a.box);
      double r2 = dadd(dadd(dmul(r[0], r[0]), dmul(r[1], r[1])), dmul(r[2], r[2]));
      return r2 > a.rc2 ? 0 : 1;
    }
    double h = ldexp(a.h0, -(int)a.leaf_depth[j]);
    return d2_aabb(xi, c, h, a.box, 0) > a.rc2 ? 0 : 1;
  }
  double h = ldexp(a.h0, -(int)a.depth[node]);
  if (d2_aabb(xi, c, h, a.box, a.periodic) > a.rc2) return 0;
  double d[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[k] = dsub(c[k], xi[k]);
    if (a.periodic) d[k] = minimum_image(d[k], a.box);
  }
  double d2 = dadd(dadd(dmul(d[0], d[0]), dmul(d[1], d[1])), dmul(d[2], d[2]));
  return d2 > 1e-30 ? 1 : 2;
}

__device__ __forceinline__ void defer(const WalkArgs& a, uint32_t p, uint32_t node) {
  uint32_t slot = atomicAdd(a.ndeferred, 1u);
  if (slot < a.cap_deferred) a.deferred[slot] = make_uint2(p, node);
  else atomicOr(a.err, DEV_ERR_DEFERRED);
}

// FP32 pair term: m * erfc(x) / r^3 (walk units), x = r/(sqrt2 r_s), for two
// entries at once.  K_POLY: erfc as 2^P(r), the fitted polynomial of WalkArgs;
// K_AS: the A&S 7.1.26 form itself; K_ACC: the A&S form plus the Gaussian term
// (2x/sqrt(pi)) exp(-x^2) of the accurate mode.
enum { K_POLY = 0, K_AS = 1, K_ACC = 2 };
template <int KERNEL>
__device__ __forceinline__ f32x2 pair_factor2(const WalkArgs& a, f32x2 r2b, f32x2 m) {
  const f32x2 r2 = add2(r2b, a.eps2_2);
  const float2 q = unpack2(r2);
  const f32x2 ri = pack2(rsqrt_approx(q.x), rsqrt_approx(q.y));
  const f32x2 r = mul2(r2, ri);
  const f32x2 ri3 = mul2(mul2(ri, ri), ri);
  f32x2 w;
  if (KERNEL == K_POLY) {
    // The coefficients stay in the constant bank: held in registers (over a
    // list) they slow the walk from 40.3 to 45.0 ms at 256^3, three 64-bit
    // register operands being more than a packed FMA reads per cycle.
    f32x2 p = a.poly2[POLY_DEGREE];
#pragma unroll
    for (int k = POLY_DEGREE - 1; k >= 0; --k) p = fma2(p, r, a.poly2[k]);
    const float2 e = unpack2(p);
    w = pack2(ex2_approx(e.x), ex2_approx(e.y));
  } else {
    const float2 d = unpack2(fma2(pack2(a.pcx, a.pcx), r, pack2(1.f, 1.f)));
    const f32x2 t = pack2(rcp_approx(d.x), rcp_approx(d.y));
    f32x2 p = pack2(ErfcConst::A5, ErfcConst::A5);
    p = fma2(p, t, pack2(ErfcConst::A4, ErfcConst::A4));
    p = fma2(p, t, pack2(ErfcConst::A3, ErfcConst::A3));
    p = fma2(p, t, pack2(ErfcConst::A2, ErfcConst::A2));
    p = fma2(p, t, pack2(ErfcConst::A1, ErfcConst::A1));
    p = mul2(p, t);
    if (KERNEL == K_ACC) p = fma2(pack2(a.gkc, a.gkc), r, p);
    const float2 e = unpack2(mul2(r2, pack2(a.ex2k, a.ex2k)));
    w = mul2(p, pack2(ex2_approx(e.x), ex2_approx(e.y)));
  }
  return mul2(mul2(m, w), ri3);
}
template <int KERNEL>
__device__ __forceinline__ float pair_factor(const WalkArgs& a, float r2b, float m) {
  return unpack2(pair_factor2<KERNEL>(a, pack2(r2b, r2b), pack2(m, m))).x;
}

struct Acc {
  float sx, sy, sz, cx, cy, cz;  // Kahan sums and compensations
  __device__ void add(float x, float y, float z) {
    float t, v;
    v = x - cx; t = sx + v; cx = (t - sx) - v; sx = t;
    v = y - cy; t = sy + v; cy = (t - sy) - v; sy = t;
    v = z - cz; t = sz + v; cz = (t - sz) - v; sz = t;
  }
};

// Lanes of the pair phase.  A group of c targets leaves 32 - c lanes without
// a target of their own, so R = 32 / c lanes share each target: lane l
// evaluates target l % c against the entry pairs l / c, l / c + R, ... of each
// list (lanes from R c on evaluate nothing), and the R partial sums of a target
// are folded when its walk ends.  Packed in one register: target | first
// pair << 8 | R << 16.
__device__ __forceinline__ uint32_t pair_lanes(int lane, uint32_t c) {
  const uint32_t r = 32u / c, t = (uint32_t)lane % c, off = (uint32_t)lane / c;
  return t | ((off < r ? off : 255u) << 8) | (r << 16);
}

// How a list's entries are cut at r_cut: on their bare distance (leaves of the
// periodic walk), or on the gap to their box of one half side for the whole
// list (monopoles of the parity walk: all at the terminal depth) or of their
// own half sides (accurate monopoles, leaves of the aperiodic walk).
enum { CUT_BARE = 0, CUT_ONE_HALF = 1, CUT_OWN_HALF = 2 };

struct Sums {
  float x, y, z;
  uint32_t n;  // entries taken
};

template <int CUT>
__device__ __forceinline__ float cut_s(float dx, float dy, float dz, float r2b, float h) {
  if (CUT == CUT_BARE) return r2b;
  const float ex = fmaxf(fabsf(dx) - h, 0.f), ey = fmaxf(fabsf(dy) - h, 0.f), ez = fmaxf(fabsf(dz) - h, 0.f);
  return fmaf(ex, ex, fmaf(ey, ey, ez * ez));
}

// One lane's share of a list, two entries per iteration in packed arithmetic
// (issue slots bound the walk, and the f32x2 instructions halve those of the
// distance, the polynomial and the sums).  Returns true when the lane met a
// pair that the loop cannot settle: one inside the band around r_cut^2 or (NEAR)
// one at a distance^2 below near.  Its result is then void, and redo_lane
// evaluates the lane's share again.  So the loop itself keeps only the
// sign of s - r_cut^2 and two running minima per pair of entries.
template <int CUT, bool BAND, bool NEAR, bool OWN, int KERNEL, class L>
__device__ __forceinline__ bool eval_list(const WalkArgs& a, const L& list, int n, uint32_t lanes, float tx, float ty,
                                          float tz, float near, Sums& out) {
  const uint32_t tbit = 1u << (lanes & 0xffu);
  const uint32_t stride = lanes >> 16;
  auto* e = &list.pair[(lanes >> 8) & 0xffu];
  const auto* end = &list.pair[(n + 1) >> 1];
  const f32x2 ntx = pack2(-tx, -tx), nty = pack2(-ty, -ty), ntz = pack2(-tz, -tz);
  const f32x2 nmid = pack2(-a.prc2_mid, -a.prc2_mid);
  f32x2 fx = 0ull, fy = 0ull, fz = 0ull;
  uint32_t cnt = 0;
  float edge = 1e30f, close = 1e30f;
#pragma unroll 1
  for (; e < end; e += stride) {
    const float4 A = e->xy, B = e->zm;
    const uint2 M = e->mask;
    const f32x2 dx = add2(pack2(A.x, A.y), ntx), dy = add2(pack2(A.z, A.w), nty), dz = add2(pack2(B.x, B.y), ntz);
    const f32x2 r2b = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    f32x2 s = r2b;
    if (CUT != CUT_BARE) {
      float2 h = make_float2(a.h_term, a.h_term);
      if constexpr (CUT == CUT_OWN_HALF) h = e->h;
      const float2 x = unpack2(dx), y = unpack2(dy), z = unpack2(dz);
      const f32x2 ex = pack2(fmaxf(fabsf(x.x) - h.x, 0.f), fmaxf(fabsf(x.y) - h.y, 0.f));
      const f32x2 ey = pack2(fmaxf(fabsf(y.x) - h.x, 0.f), fmaxf(fabsf(y.y) - h.y, 0.f));
      const f32x2 ez = pack2(fmaxf(fabsf(z.x) - h.x, 0.f), fmaxf(fabsf(z.y) - h.y, 0.f));
      s = fma2(ex, ex, fma2(ey, ey, mul2(ez, ez)));
    }
    const float2 q = unpack2(add2(s, nmid));
    if (BAND) edge = min3_abs(edge, q.x, q.y);
    const bool in0 = M.x & tbit, in1 = M.y & tbit;
    if (NEAR) {  // (OWN: the target's own leaf, at no distance, is not for it to see)
      const float2 c = unpack2(r2b);
      close = OWN ? min3_abs(close, in0 ? c.x : 1e30f, in1 ? c.y : 1e30f) : min3_abs(close, c.x, c.y);
    }
    const bool ok0 = in0 && q.x <= 0.f, ok1 = in1 && q.y <= 0.f;
    const float2 f = unpack2(pair_factor2<KERNEL>(a, r2b, pack2(B.z, B.w)));
    const f32x2 g = pack2(ok0 ? f.x : 0.f, ok1 ? f.y : 0.f);
    fx = fma2(dx, g, fx);
    fy = fma2(dy, g, fy);
    fz = fma2(dz, g, fz);
    cnt += ok0 ? 1u : 0u;  // the target's own leaf is masked out at emission
    cnt += ok1 ? 1u : 0u;
  }
  const float2 X = unpack2(fx), Y = unpack2(fy), Z = unpack2(fz);
  out.x = X.x + X.y;
  out.y = Y.x + Y.y;
  out.z = Z.x + Z.y;
  out.n = cnt;
  return (BAND && edge <= a.pband) || (NEAR && close < near);
}

// Position of a list entry's source, in quanta.
__device__ __forceinline__ void source_quanta(const WalkArgs& a, uint32_t node, uint32_t q[3]) {
  if (node & LEAF_BIT) {
    const uint32_t j = node & ~LEAF_BIT;
    q[0] = a.qx[j];
    q[1] = a.qy[j];
    q[2] = a.qz[j];
  } else {
    const uint4 w = a.walk[node];
    q[0] = w.x;
    q[1] = w.y;
    q[2] = w.z;
  }
}

// The share of lane `src` again (rare), all 32 lanes taking entry pairs of it,
// with the reference's float64 decisions for the undecided entries (MONO: also
// for a centre of mass within a few quanta of the target) and, CLOSE, the exact
// coordinate differences for the near ones.  Every lane returns the sums.
template <int CUT, bool BAND, bool MONO, bool CLOSE, bool PERIODIC, int KERNEL, class L>
__device__ __noinline__ Sums redo_lane(const WalkArgs& a, const L& list, int n, uint32_t lanes, uint32_t p, float tx,
                                       float ty, float tz, float near, uint32_t* nexact) {
  const int t = lanes & 0xffu, stride = lanes >> 16, lane = threadIdx.x & 31;
  Sums o = {0.f, 0.f, 0.f, 0u};
  for (int e = 2 * (int)(((lanes >> 8) & 0xffu) + (uint32_t)(lane * stride)); e < n; e += 64 * stride) {
    for (int k = e; k < e + 2 && k < n; ++k) {
      const float* w = list.word(k);
      const uint32_t node = __float_as_uint(w[10]);
      if (!((__float_as_uint(w[8]) >> t) & 1u)) continue;
      float dx = w[0] - tx, dy = w[2] - ty, dz = w[4] - tz;
      float r2b = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      if (CLOSE && r2b < near) {
        uint32_t q[3];
        source_quanta(a, node, q);
        dx = rel(q[0], a.qx[p], PERIODIC) * a.u_inv;
        dy = rel(q[1], a.qy[p], PERIODIC) * a.u_inv;
        dz = rel(q[2], a.qz[p], PERIODIC) * a.u_inv;
        r2b = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      }
      const float s = cut_s<CUT>(dx, dy, dz, r2b, CUT == CUT_OWN_HALF ? w[12] : a.h_term);
      bool take = s <= a.prc2_lo;
      if (BAND && ((s > a.prc2_lo && s <= a.prc2_hi) || (MONO && r2b < a.tiny_u))) {
        ++*nexact;
        const int d = exact_terminal(a, p, node);
        if (d == 2) defer(a, p, node);
        take = d == 1;
      }
      if (!take) continue;
      const float f = pair_factor<KERNEL>(a, r2b, w[6]);
      o.x = fmaf(dx, f, o.x);
      o.y = fmaf(dy, f, o.y);
      o.z = fmaf(dz, f, o.z);
      ++o.n;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    o.x += __shfl_xor_sync(0xffffffffu, o.x, off);
    o.y += __shfl_xor_sync(0xffffffffu, o.y, off);
    o.z += __shfl_xor_sync(0xffffffffu, o.z, off);
    o.n += __shfl_xor_sync(0xffffffffu, o.n, off);
  }
  return o;
}

// A list against this lane's pair-phase target (its position comes from the
// lane that holds it, its particle is first + target).
template <int CUT, bool MONO, bool CLOSE, bool PERIODIC, int KERNEL, class L>
__device__ __forceinline__ Sums eval(const WalkArgs& a, const L& list, int n, uint32_t lanes, uint32_t first,
                                     const float4* tfs, const float4& T, float near, uint32_t& nexact) {
  // (the accurate mode reproduces no float64 decisions)
  constexpr bool BAND = KERNEL != K_ACC, NEAR = CLOSE || (MONO && BAND);
  Sums o;
  const bool flag = eval_list<CUT, BAND, NEAR, !MONO, KERNEL>(a, list, n, lanes, T.x, T.y, T.z, near, o);
  if (BAND || NEAR) {
    uint32_t again = __ballot_sync(0xffffffffu, flag);
    while (again) {
      const int src = __ffs(again) - 1;
      again &= again - 1;
      const uint32_t sl = __shfl_sync(0xffffffffu, lanes, src);
      const float4 S = tfs[sl & 0xffu];
      const Sums r = redo_lane<CUT, BAND, MONO, CLOSE, PERIODIC, KERNEL>(a, list, n, sl, first + (sl & 0xffu), S.x, S.y,
                                                                         S.z, near, &nexact);
      if ((threadIdx.x & 31) == src) o = r;
    }
  }
  return o;
}

// Evaluate both interaction lists against this lane's pair-phase target.
// The lane's running sums live in shared memory between flushes (s0 = sx, sy,
// sz, cx; s1 = cy, cz, leaf count, monopole count bits), so they hold no
// registers across the traversal.
template <bool PERIODIC, int KERNEL> struct Lists {
  static constexpr bool ACC = KERNEL == K_ACC;
  List<chunk_l<ACC>(), !PERIODIC> leaf;
  List<chunk_m<ACC>(), ACC || !PERIODIC> mono;
};
template <bool PERIODIC, int KERNEL, bool CLOSE>
__device__ __forceinline__ void flush(const WalkArgs& a, const Lists<PERIODIC, KERNEL>& lists, int nll, int nlm,
                                      int lane, uint32_t lanes, uint32_t first, const float4* tfs, float near,
                                      float4* s0, float4* s1, uint32_t& nexact, uint32_t& neval) {
  constexpr bool ACC = KERNEL == K_ACC;
  neval += (uint32_t)(nll + nlm);
  const float4 T = tfs[lanes & 0xffu];
  const Sums l = eval<PERIODIC ? CUT_BARE : CUT_OWN_HALF, false, CLOSE, PERIODIC, KERNEL>(a, lists.leaf, nll, lanes,
                                                                                          first, tfs, T, near, nexact);
  const Sums m = eval<ACC ? CUT_OWN_HALF : CUT_ONE_HALF, true, CLOSE, PERIODIC, KERNEL>(a, lists.mono, nlm, lanes,
                                                                                        first, tfs, T, near, nexact);
  __syncwarp();
  const float4 A = s0[lane], B = s1[lane];
  Acc acc = {A.x, A.y, A.z, A.w, B.x, B.y};
  acc.add(l.x + m.x, l.y + m.y, l.z + m.z);
  s0[lane] = make_float4(acc.sx, acc.sy, acc.sz, acc.cx);
  s1[lane] = make_float4(acc.cy, acc.cz, __uint_as_float(__float_as_uint(B.z) + l.n),
                         __uint_as_float(__float_as_uint(B.w) + m.n));
}

// CLOSE: pairs nearer than a sixteenth of the group's extent take their exact
// coordinate differences (in distance^2, over the square of half the extent).  A
// relative position is off by up to 2^-25 of half the extent, so a pair beyond
// that keeps its distance to 5e-7 per coordinate, and the nearer ones are few:
// walk of 32^3 particles .203 -> .208 ms, 48^3 .410 -> .418 (at an eighth .210
// and .440), error of the short range against float64 in four boxes of 32^3
// 4.3 .. 5.5e-7 -> 2.2 .. 2.5e-7 (1.9 .. 2.4e-7), of 48^3 3.5 .. 6.8e-7 -> 2.6 .. 2.8e-7.
constexpr float NEAR_SHARE = 1.f / 64.f;

constexpr int STACK_ENTRIES = 1024;  // global, per warp

// End of a group's walk: fold the pair-phase lanes of each target, write its
// acceleration and interaction counts, add to the statistics.
__device__ __forceinline__ void store_sums(const WalkArgs& a, uint32_t p, bool has, uint32_t count, float4 S0,
                                           float4 S1, uint32_t nexact, uint32_t neval) {
  const int lane = threadIdx.x & 31;
  Acc acc = {S0.x, S0.y, S0.z, S0.w, S1.x, S1.y};
  uint32_t nleaf = __float_as_uint(S1.z), nmono = __float_as_uint(S1.w);
  // fold the R pair-phase lanes of each target (lanes t + j count) into lane t
  const uint32_t nrep = 32u / count;
  for (uint32_t j = 1; j < nrep; ++j) {
    const int src = lane + (int)(j * count);  // in range for the lanes t < count that keep the result
    const float ox = __shfl_sync(0xffffffffu, acc.sx, src), oy = __shfl_sync(0xffffffffu, acc.sy, src);
    const float oz = __shfl_sync(0xffffffffu, acc.sz, src);
    const float cx = __shfl_sync(0xffffffffu, acc.cx, src), cy = __shfl_sync(0xffffffffu, acc.cy, src);
    const float cz = __shfl_sync(0xffffffffu, acc.cz, src);
    const uint32_t ol = __shfl_sync(0xffffffffu, nleaf, src), om = __shfl_sync(0xffffffffu, nmono, src);
    if ((uint32_t)lane < count) {
      acc.add(ox - cx, oy - cy, oz - cz);
      nleaf += ol;
      nmono += om;
    }
  }
  if (has) {
    a.ax[p] = (acc.sx - acc.cx) * a.out_scale;
    a.ay[p] = (acc.sy - acc.cy) * a.out_scale;
    a.az[p] = (acc.sz - acc.cz) * a.out_scale;
    a.pcounts[2 * (int64_t)p] = nleaf;
    a.pcounts[2 * (int64_t)p + 1] = nmono;
  }
  if ((uint32_t)lane >= count) nleaf = nmono = 0;  // counted once per target
  // statistics
  unsigned long long l = nleaf, m = nmono, x = nexact;
  for (int off = 16; off > 0; off >>= 1) {
    l += __shfl_down_sync(0xffffffffu, l, off);
    m += __shfl_down_sync(0xffffffffu, m, off);
    x += __shfl_down_sync(0xffffffffu, x, off);
  }
  if (lane == 0) {
    atomicAdd(&a.stats[0], l);
    atomicAdd(&a.stats[1], m);
    atomicAdd(&a.stats[2], (unsigned long long)neval * 32ull / nrep);  // lane evaluations
    atomicAdd(&a.stats[3], x);
  }
}

// Shared memory of one warp.
template <bool PERIODIC, int KERNEL> struct __align__(16) WarpMem {
  static constexpr bool ACC = KERNEL == K_ACC;
  Lists<PERIODIC, KERNEL> lists;
  // undecided nodes of an open step (their cull half side in place of the
  // mass; accurate: their half side as well), the targets that go on to their
  // children and (accurate) those that take them as monopoles
  List<32, ACC> nodes;
  uint32_t seen[32];
  uint32_t taken[ACC ? 32 : 4];
  float4 cells[ACC ? 32 : 1];  // relative criterion: cell centre, |Q|_F / M of the undecided nodes
  float4 s0[32], s1[32];       // the lanes' running sums
  float4 tfs[32];              // target positions
  float4 gbox[2];              // half widths of the group box and the near distance^2, the origin
  uint4 queue[40];             // nodes whose terminal children wait {first record, count, mask}
};

// The opening decision of the accurate mode for a target at distance^2 d2 from
// the centre of mass of a node of half side h: the opening angle s/d < theta,
// s = 2 h (octree.rs:763-809).
__device__ __forceinline__ bool accept_angle(const WalkArgs& a, float h, float d2) {
  return 4.f * h * h < a.theta2 * d2;
}
// Relative criterion (octree.rs:769-796), qm = |Q|_F / M: the truncation
// estimate |Q|_F (d^2 + eps^2) < k M d^5 (the caller checks that the target is
// outside the node's cell).
__device__ __forceinline__ bool accept_relative(const WalkArgs& a, float qm, float d2, float margin) {
  return d2 > 0.f && qm * (d2 + a.eps2_u) < a.rel_k * (d2 * d2 * sqrtf(d2)) * margin;
}

// The staged undecided nodes of an open step, one at a time: where a node is
// seen at another periodic image by part of the group (marked in its node
// word), a target lies inside the band around r_cut^2 (parity: the reference's
// float64 test decides), or the relative criterion opens nodes.
template <bool PERIODIC, int KERNEL>
__device__ __noinline__ uint32_t refine_slow(const WalkArgs& a, WarpMem<PERIODIC, KERNEL>& mem, int n, uint32_t p,
                                             float4 T) {
  constexpr bool ACC = KERNEL == K_ACC;
  const int lane = threadIdx.x & 31;
  uint32_t nexact = 0;
  for (int j = 0; j < n; ++j) {
    const float* w = mem.nodes.word(j);
    const uint32_t node = __float_as_uint(w[10]);
    float dx = w[0] - T.x, dy = w[2] - T.y, dz = w[4] - T.z;
    if (PERIODIC && (node & LEAF_BIT)) {
      dx -= a.box_u * rintf(dx / a.box_u);
      dy -= a.box_u * rintf(dy / a.box_u);
      dz -= a.box_u * rintf(dz / a.box_u);
    }
    const float s = cut_s<CUT_OWN_HALF>(dx, dy, dz, 0.f, w[6]);
    const bool in = (__float_as_uint(w[8]) >> lane) & 1u;
    bool pass = in && s <= a.rc2_lo, take = false;
    if (!ACC && in && !pass && s <= a.rc2_hi) {
      pass = exact_open_pass(a, p, node & ~LEAF_BIT);
      ++nexact;
    }
    if (ACC && pass) {
      const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz)), h = fabsf(w[12]);
      if (!a.relative) {
        take = accept_angle(a, h, d2);
      } else if (w[12] > 0.f) {  // (nodes of the top levels are always opened)
        // point_in_node_cell with a margin: a target on the cell's face opens the node
        const float4 C = mem.cells[j];
        float cx = C.x - T.x, cy = C.y - T.y, cz = C.z - T.z;
        const bool inside = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) <= h * 1.0001f;
        take = !inside && accept_relative(a, C.w, d2, 1.f);
      }
    }
    const uint32_t tm = ACC ? __ballot_sync(0xffffffffu, take) : 0u;
    const uint32_t nm = __ballot_sync(0xffffffffu, pass) & ~tm;
    if (lane == 0) {
      mem.seen[j] = nm;
      if (ACC) mem.taken[j] = tm;
    }
  }
  return nexact;
}

// Walk of targets [first, first + count) (count <= 32) with one warp.
//
// An octree node's children are stored internal nodes first, leaves after
// them.  Parity: internal nodes become monopoles at one depth for the whole
// tree; accurate: where a target's distance allows it.  So a node that stays
// open splits into a range of open children and a range of terminal ones, and
// the walk has two kinds of step, each on four nodes at a time with eight lanes
// per node (a node has at most eight children, so no lane has to look up its
// child): an open step classifies open children against the group box, tests
// the undecided ones per target and pushes what is seen; an item step cuts
// terminal children against the group box and appends them to the lists.  The
// item step, which meets most of the nodes, needs neither the periodic images
// nor the opening test.
template <bool PERIODIC, int KERNEL, bool CLOSE>
__device__ __forceinline__ void walk_group(const WalkArgs& a, uint32_t first, uint32_t count,
                                           WarpMem<PERIODIC, KERNEL>& mem, uint4* stk) {
  constexpr bool ACC = KERNEL == K_ACC;
  const int lane = threadIdx.x & 31;
  const uint32_t p = first + ((uint32_t)lane < count ? (uint32_t)lane : 0u);
  // targets of this walk: the group's particles, or those of them the caller
  // selected (the group box then covers only those)
  const bool has = (uint32_t)lane < count && (!a.only || a.only[p] != 0);
  const uint32_t mask0 = __ballot_sync(0xffffffffu, has);  // bit t: target t
  if (mask0 == 0u) return;
  const int term_depth = ACC ? 64 : a.term_depth;
  {
    const uint32_t tq[3] = {a.qx[p], a.qy[p], a.qz[p]};
    uint32_t oq[3];
    float tf[3], w[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      // positions relative to the middle of the group's box: half the extent
      // bounds them, and with them the rounding of the pair distances
      const uint32_t q0 = __shfl_sync(0xffffffffu, tq[d], 0);
      // (a group lies in a cell far smaller than half the box)
      const int32_t tr = (int32_t)(tq[d] - q0);
      const int32_t lo = __reduce_min_sync(0xffffffffu, has ? tr : 0x7FFFFFFF);
      const int32_t hi = __reduce_max_sync(0xffffffffu, has ? tr : -0x7FFFFFFF);
      const int32_t mid = lo + ((hi - lo) >> 1);
      oq[d] = q0 + (uint32_t)mid;
      tf[d] = (float)(tr - mid) * a.u_inv;
      w[d] = (float)(hi - mid) * a.u_inv;
    }
    mem.tfs[lane] = make_float4(tf[0], tf[1], tf[2], 0.f);
    if (lane == 0) {
      const float wide = fmaxf(w[0], fmaxf(w[1], w[2]));  // half the group's extent
      mem.gbox[0] = make_float4(w[0], w[1], w[2], CLOSE ? fmaxf(a.tiny_u, NEAR_SHARE * wide * wide) : a.tiny_u);
      reinterpret_cast<uint4*>(mem.gbox)[1] = make_uint4(oq[0], oq[1], oq[2], 0u);
      // the root: a terminal node by itself, or an open one
      if (term_depth == 0) mem.queue[0] = make_uint4(0u, 1u, mask0, 0u);
      else stk[0] = make_uint4(0u, 1u, mask0, 0u);
    }
  }
  mem.s0[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  mem.s1[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  const uint32_t lanes = pair_lanes(lane, count);
  uint32_t nexact = 0, neval = 0;
  int nll = 0, nlm = 0, sp = term_depth == 0 ? 0 : 1, nq = 1 - sp;
  // each step takes at least one range, and a node makes at most two: the cap
  // turns a malformed tree into an error flag instead of an endless loop
  uint32_t steps_left = (uint32_t)(2 * a.n_int + 4 < 0xFFFFFFFFll ? 2 * a.n_int + 4 : 0xFFFFFFFFll);
  const uint32_t below = (1u << lane) - 1u;
  __syncwarp();
  const int slot = lane >> 3, child = lane & 7;
  for (;;) {
    // a step adds up to 32 entries to either list (one call site of the list
    // evaluation, the last flush included)
    const bool done = sp == 0 && nq == 0;
    if (done || nll > chunk_l<ACC>() - 32 || nlm > chunk_m<ACC>() - 32) {
      if (lane == 0) {
        mem.lists.leaf.close(nll);
        mem.lists.mono.close(nlm);
      }
      __syncwarp();
      flush<PERIODIC, KERNEL, CLOSE>(a, mem.lists, nll, nlm, lane, lanes, first, mem.tfs, mem.gbox[0].w, mem.s0, mem.s1,
                                     nexact, neval);
      __syncwarp();
      nll = 0;
      nlm = 0;
      if (done) break;
    }
    if (steps_left-- == 0u) {
      if (lane == 0) atomicOr(a.err, DEV_ERR_STACK);
      break;
    }
    const float4 GW = mem.gbox[0];
    const uint4 GO = reinterpret_cast<const uint4*>(mem.gbox)[1];
    if (nq >= 4 || sp == 0) {  // ---- item step
      const int np = nq < 4 ? nq : 4;
      uint4 e = make_uint4(0u, 0u, 0u, 0u);
      if (slot < np) e = mem.queue[nq - 1 - slot];
      nq -= np;
      bool keep = (uint32_t)child < e.y;
      uint4 r0 = make_uint4(0u, 0u, 0u, 0u), r1 = r0;
      if (keep) {
        const uint4* rec = reinterpret_cast<const uint4*>(&a.recs[e.x + (uint32_t)child]);
        r0 = __ldg(rec);
        r1 = __ldg(rec + 1);
      }
      const bool leaf = ACC || (r1.y & WN_LEAF) != 0u;
      const float h = !leaf ? a.h_term : (PERIODIC ? 0.f : half_side(a.h0_u, wn_depth(r1.y)));
      const float sx = rel(r0.x, GO.x, PERIODIC) * a.u_inv, sy = rel(r0.y, GO.y, PERIODIC) * a.u_inv;
      const float sz = rel(r0.z, GO.z, PERIODIC) * a.u_inv;
      // the gap between the group box and the node's box
      const float gx = fmaxf(fabsf(sx) - (GW.x + h), 0.f), gy = fmaxf(fabsf(sy) - (GW.y + h), 0.f);
      const float gz = fmaxf(fabsf(sz) - (GW.z + h), 0.f);
      keep = keep && !(fmaf(gx, gx, fmaf(gy, gy, gz * gz)) > a.grc2_hi);
      const uint32_t el = __ballot_sync(0xffffffffu, keep && leaf);
      const uint32_t em = ACC ? 0u : __ballot_sync(0xffffffffu, keep && !leaf);
      if (keep) {
        // the reference skips the target's own leaf (j != skip)
        const uint32_t own = leaf ? r1.z - first : 32u;
        const uint32_t see = own < count ? (e.z & ~(1u << own)) : e.z;
        if constexpr (ACC) {
          mem.lists.leaf.put(nll + __popc(el & below), sx, sy, sz, __uint_as_float(r0.w), h, see, r1.z | LEAF_BIT);
        } else {
          // both lists have the same layout of pairs
          List<2, !PERIODIC>::put(leaf ? mem.lists.leaf.pair : mem.lists.mono.pair,
                                  leaf ? nll + __popc(el & below) : nlm + __popc(em & below), sx, sy, sz,
                                  __uint_as_float(r0.w), h, see, leaf ? r1.z | LEAF_BIT : r1.z);
        }
      }
      nll += __popc(el);
      nlm += __popc(em);
      __syncwarp();
      continue;
    }
    // ---- open step
    const int np = sp < 4 ? sp : 4;
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    if (slot < np) e = stk[sp - 1 - slot];
    sp -= np;
    const bool live = (uint32_t)child < e.y;
    uint4 r0 = make_uint4(0u, 0u, 0u, 0u), r1 = r0;
    if (live) {
      const uint4* rec = reinterpret_cast<const uint4*>(&a.recs[e.x + (uint32_t)child]);
      r0 = __ldg(rec);
      r1 = __ldg(rec + 1);
    }
    const int dep = wn_depth(r1.y);
    const float hnode = half_side(a.h0_u, dep);
    // cull half side: the COM-centred AABB's, or (accurate) twice that, which
    // holds the whole cell
    const float h = ACC ? 2.f * hnode : hnode;
    const float sx = rel(r0.x, GO.x, PERIODIC) * a.u_inv, sy = rel(r0.y, GO.y, PERIODIC) * a.u_inv;
    const float sz = rel(r0.z, GO.z, PERIODIC) * a.u_inv;
    const float ux = fabsf(sx), uy = fabsf(sy), uz = fabsf(sz);
    // the nearest and the farthest a target can be from the node's box
    const float gx = fmaxf(ux - (GW.x + h), 0.f), gy = fmaxf(uy - (GW.y + h), 0.f), gz = fmaxf(uz - (GW.z + h), 0.f);
    const float fx = fmaxf(ux + (GW.x - h), 0.f), fy = fmaxf(uy + (GW.y - h), 0.f), fz = fmaxf(uz + (GW.z - h), 0.f);
    // Nodes that part of the group sees at another periodic image are left to
    // the per-target test, if they are wide enough for that image to come
    // within r_cut.  The others: seen by the whole group, or undecided.
    const float half_box = 0.5f * a.box_u;
    const bool top = PERIODIC && dep < a.img_depth;
    const bool image = top && live && (ux + GW.x > half_box || uy + GW.y > half_box || uz + GW.z > half_box);
    bool keep = live && (image || !(fmaf(gx, gx, fmaf(gy, gy, gz * gz)) > a.grc2_hi));
    bool ambig = keep && (image || !(fmaf(fx, fx, fmaf(fy, fy, fz * fz)) < a.grc2_lo));
    uint32_t see = e.z, take = 0u;  // targets that open the node, that take it as a monopole
    float4 cell = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ACC && keep && !image) {
      // opening test for the whole group by its nearest and farthest distances
      // from the centre of mass (both criteria are monotone in it), with a
      // margin that leaves the float-rounding cases to the per-target test
      const float nx = fmaxf(ux - GW.x, 0.f), ny = fmaxf(uy - GW.y, 0.f), nz = fmaxf(uz - GW.z, 0.f);
      const float ox = ux + GW.x, oy = uy + GW.y, oz = uz + GW.z;
      const float dmin2 = fmaf(nx, nx, fmaf(ny, ny, nz * nz)), dmax2 = fmaf(ox, ox, fmaf(oy, oy, oz * oz));
      bool all, none;
      if (a.relative) {
        // the target must be outside the node's cell: a group box touching the
        // cell leaves the node to the per-target test
        const uint4 cc = __ldg(&a.cellq[r1.z]);
        cell = make_float4(rel(cc.x, GO.x, PERIODIC) * a.u_inv, rel(cc.y, GO.y, PERIODIC) * a.u_inv,
                           rel(cc.z, GO.z, PERIODIC) * a.u_inv, __uint_as_float(cc.w) / __uint_as_float(r0.w));
        const float hc = hnode * 1.0001f;
        const bool touch = fabsf(cell.x) <= GW.x + hc && fabsf(cell.y) <= GW.y + hc && fabsf(cell.z) <= GW.z + hc;
        const bool inside = fabsf(cell.x) + GW.x <= hc && fabsf(cell.y) + GW.y <= hc && fabsf(cell.z) + GW.z <= hc;
        none = top || inside || !accept_relative(a, cell.w, dmax2, 1.001f);
        all = !none && !touch && accept_relative(a, cell.w, dmin2, 0.999f);
      } else {
        all = accept_angle(a, hnode, dmin2 * 0.999f);
        none = !accept_angle(a, hnode, dmax2 * 1.001f);
      }
      if (all) {  // the pair loop cuts it per target
        take = e.z;
        see = 0u;
        ambig = false;
      } else {
        ambig = ambig || !none;
      }
    }
    const uint32_t amb = __ballot_sync(0xffffffffu, ambig);
    if (amb != 0u) {
      // Per-target refinement: each undecided node is staged once in shared
      // memory, then tested against all targets (one per lane), two nodes at a
      // time in packed arithmetic.  dd = COM - target in float differs from
      // the exact minimum-image difference by ~1e-7 of r_cut, far inside the
      // band around r_cut^2 that goes to the float64 test.
      const int mine = __popc(amb & below), namb = __popc(amb);
      if (ambig) {
        mem.nodes.put(mine, sx, sy, sz, h, top ? -hnode : hnode, e.z, image ? r1.z | LEAF_BIT : r1.z);
        if (ACC && a.relative) mem.cells[mine] = cell;
      }
      if (lane == 0) mem.nodes.close(namb);
      bool slow = __any_sync(0xffffffffu, image) || (ACC && a.relative);
      __syncwarp();
      const float4 TF = mem.tfs[lane];
      if (!slow) {
        const f32x2 ntx = pack2(-TF.x, -TF.x), nty = pack2(-TF.y, -TF.y), ntz = pack2(-TF.z, -TF.z);
        const uint32_t tbit = 1u << lane;
        float edge = 1e30f;
        const f32x2 nmid = pack2(-a.rc2_mid, -a.rc2_mid);
        for (int j = 0; j < namb; j += 2) {
          auto& nd = mem.nodes.pair[j >> 1];
          const float4 A = nd.xy, B = nd.zm;
          const uint2 M = nd.mask;
          const f32x2 dx = add2(pack2(A.x, A.y), ntx), dy = add2(pack2(A.z, A.w), nty);
          const f32x2 dz = add2(pack2(B.x, B.y), ntz);
          const float2 x = unpack2(dx), y = unpack2(dy), z = unpack2(dz);
          const f32x2 ex = pack2(fmaxf(fabsf(x.x) - B.z, 0.f), fmaxf(fabsf(x.y) - B.w, 0.f));
          const f32x2 ey = pack2(fmaxf(fabsf(y.x) - B.z, 0.f), fmaxf(fabsf(y.y) - B.w, 0.f));
          const f32x2 ez = pack2(fmaxf(fabsf(z.x) - B.z, 0.f), fmaxf(fabsf(z.y) - B.w, 0.f));
          const float2 q = unpack2(add2(fma2(ez, ez, fma2(ey, ey, mul2(ex, ex))), nmid));
          const bool p0 = (M.x & tbit) && q.x <= 0.f, p1 = (M.y & tbit) && q.y <= 0.f;
          uint32_t n0 = __ballot_sync(0xffffffffu, p0), n1 = __ballot_sync(0xffffffffu, p1);
          if constexpr (ACC) {
            const float2 d2 = unpack2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)))), hn = nd.h;
            const uint32_t t0 = __ballot_sync(0xffffffffu, p0 && accept_angle(a, hn.x, d2.x));
            const uint32_t t1 = __ballot_sync(0xffffffffu, p1 && accept_angle(a, hn.y, d2.y));
            n0 &= ~t0;
            n1 &= ~t1;
            if (lane == 0) *reinterpret_cast<uint2*>(&mem.taken[j]) = make_uint2(t0, t1);
          } else {
            edge = min3_abs(edge, q.x, q.y);
          }
          if (lane == 0) *reinterpret_cast<uint2*>(&mem.seen[j]) = make_uint2(n0, n1);
        }
        if (!ACC) slow = __any_sync(0xffffffffu, edge <= a.rc2_band);
      }
      if (slow) nexact += refine_slow<PERIODIC, KERNEL>(a, mem, namb, p, TF);
      __syncwarp();
      if (ambig) {
        see = mem.seen[mine];
        if (ACC) take = mem.taken[mine];
      }
    }
    if constexpr (ACC) {
      const uint32_t em = __ballot_sync(0xffffffffu, keep && take != 0u);
      if (keep && take != 0u)
        mem.lists.mono.put(nlm + __popc(em & below), sx, sy, sz, __uint_as_float(r0.w), h, take, r1.z);
      nlm += __popc(em);
    }
    keep = keep && see != 0u;  // a node no target opens is not pushed
    // the seen nodes' children: internal ones stay open above the terminal
    // depth, the rest are items
    const uint32_t inner = dep + 1 < term_depth ? wn_ninner(r1.y) : 0u, rest = wn_nchild(r1.y) - inner;
    const uint32_t po = __ballot_sync(0xffffffffu, keep && inner != 0u);
    const uint32_t pi = __ballot_sync(0xffffffffu, keep && rest != 0u);
    if (sp + __popc(po) > STACK_ENTRIES) {
      if (lane == 0) atomicOr(a.err, DEV_ERR_STACK);
      break;
    }
    if (keep && inner != 0u) stk[sp + __popc(po & below)] = make_uint4(r1.x, inner, see, 0u);
    if (keep && rest != 0u) mem.queue[nq + __popc(pi & below)] = make_uint4(r1.x + inner, rest, see, 0u);
    sp += __popc(po);
    nq += __popc(pi);
    __syncwarp();
  }
  __syncwarp();
  store_sums(a, p, has, count, mem.s0[lane], mem.s1[lane], nexact, neval);
}

template <int MIN_BLOCKS, bool PERIODIC, int KERNEL, bool CLOSE>
__global__ void __launch_bounds__(WALK_THREADS, MIN_BLOCKS) k_walk(const __grid_constant__ WalkArgs a) {
  extern __shared__ __align__(16) unsigned char s_walk[];
  using Mem = WarpMem<PERIODIC, KERNEL>;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Mem& mem = reinterpret_cast<Mem*>(s_walk)[wid];
  // a list's unused half pair is evaluated and dropped: it must hold numbers
  for (int i = lane; i < (int)(sizeof(mem.lists) / sizeof(uint32_t)); i += 32)
    reinterpret_cast<uint32_t*>(&mem.lists)[i] = 0u;
  __syncwarp();
  const int64_t gw = (int64_t)blockIdx.x * WALK_WARPS + wid;
  uint4* stk = reinterpret_cast<uint4*>(a.stack) + gw * STACK_ENTRIES;
  const uint32_t ngroups = *a.ngroups;
  for (;;) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(a.work, 1u);
    g = __shfl_sync(0xffffffffu, g, 0);
    if (g >= ngroups) break;
    const uint32_t first = a.gfirst[g], count = a.gsize[g];
    walk_group<PERIODIC, KERNEL, CLOSE>(a, first, count, mem, stk);
  }
}

// ---- per-target exact walk below a node whose centre of mass coincides with
// the target (the reference opens such a monopole, short_range.rs:316-330)
__device__ void deferred_walk(const WalkArgs& a, uint2 job) {
  const uint32_t p = job.x;
  double xi[3];
  target_pos(a, p, xi);
  const uint32_t tq[3] = {a.qx[p], a.qy[p], a.qz[p]};
  uint32_t stack[8 * 48];
  int sp = 0;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  // push the children of a node
  auto open = [&](uint32_t nd) {
    for (int k = 0; k < 8; ++k) {
      const uint32_t c = a.slots[8 * (int64_t)nd + k];
      if (c != EMPTY_SLOT) stack[sp++] = c;
    }
  };
  open(job.y);
  int64_t guard = 0;
  while (sp > 0) {
    if (++guard > a.n_int + a.n + 2) {
      atomicOr(a.err, DEV_ERR_STACK);
      break;
    }
    const uint32_t node = stack[--sp];
    double c[3];
    node_com(a, node, c);
    float m;
    uint32_t cq[3];
    if (node & LEAF_BIT) {
      const uint32_t j = node & ~LEAF_BIT;
      m = a.massf[j];
      cq[0] = a.qx[j]; cq[1] = a.qy[j]; cq[2] = a.qz[j];
    } else {
      const uint4 w = a.walk[node];
      m = __uint_as_float(w.w);
      cq[0] = w.x; cq[1] = w.y; cq[2] = w.z;
    }
    const int dep = (node & LEAF_BIT) ? a.leaf_depth[node & ~LEAF_BIT] : a.depth[node];
    const double h = ldexp(a.h0, -dep);
    if (d2_aabb(xi, c, h, a.box, a.periodic) > a.rc2) continue;
    bool interact = false;
    if (node & LEAF_BIT) {
      if ((node & ~LEAF_BIT) == p) continue;
      interact = exact_terminal(a, p, node) == 1;
    } else if (h < a.thr) {
      const int d = exact_terminal(a, p, node);
      if (d == 1) interact = true;
      else if (d == 2) {
        if (sp + 8 > 8 * 48) { atomicOr(a.err, DEV_ERR_STACK); break; }
        open(node);
      }
    } else {
      if (sp + 8 > 8 * 48) { atomicOr(a.err, DEV_ERR_STACK); break; }
      open(node);
    }
    if (interact) {
      atomicAdd(&a.pcounts[2 * (int64_t)p + ((node & LEAF_BIT) ? 0 : 1)], 1u);
      const float dx = rel(cq[0], tq[0], a.periodic) * a.u_inv;
      const float dy = rel(cq[1], tq[1], a.periodic) * a.u_inv;
      const float dz = rel(cq[2], tq[2], a.periodic) * a.u_inv;
      const float r2b = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const float f = a.poly ? pair_factor<K_POLY>(a, r2b, m) : pair_factor<K_AS>(a, r2b, m);
      fx = fmaf(dx, f, fx);
      fy = fmaf(dy, f, fy);
      fz = fmaf(dz, f, fz);
    }
  }
  atomicAdd(&a.ax[p], fx * a.out_scale);
  atomicAdd(&a.ay[p], fy * a.out_scale);
  atomicAdd(&a.az[p], fz * a.out_scale);
  atomicAdd(&a.stats[4], 1ull);
}

__global__ void k_deferred(const __grid_constant__ WalkArgs a) {
  const uint32_t n = min(*a.ndeferred, a.cap_deferred);
  for (uint32_t it = blockIdx.x * blockDim.x + threadIdx.x; it < n; it += gridDim.x * blockDim.x)
    deferred_walk(a, a.deferred[it]);
}

}  // namespace

// Resident blocks (of 4 warps) per SM, i.e. the register budget: the parity
// walk takes 96 registers (clustered 256^3: 44.0 ms at 4 blocks, 40.3 at 5, 41.0
// at 6 with 72 bytes of spills), the accurate one 64 (clustered 128^3: 7.46 at 5,
// 7.40 at 6, 7.51 at 7, where shared memory leaves the L1 cache 16 KB).
template <int KERNEL> constexpr int walk_blocks() { return KERNEL == K_ACC ? 6 : 5; }

template <bool PERIODIC, int KERNEL, bool CLOSE>
static int blocks_for() {
  auto k = k_walk<walk_blocks<KERNEL>(), PERIODIC, KERNEL, CLOSE>;
  const size_t smem = sizeof(WarpMem<PERIODIC, KERNEL>) * WALK_WARPS;
  TPM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int nb = 0;
  TPM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, WALK_THREADS, smem));
  return nb < 1 ? 1 : nb;
}

template <bool PERIODIC, int KERNEL, bool CLOSE>
static void launch_t(const WalkArgs& a, int grid, cudaStream_t s) {
  const size_t smem = sizeof(WarpMem<PERIODIC, KERNEL>) * WALK_WARPS;
  k_walk<walk_blocks<KERNEL>(), PERIODIC, KERNEL, CLOSE><<<grid, WALK_THREADS, smem, s>>>(a);
}

// The kernel of a walk, by its mode, pair term and near pairs; also sizes its grid.
template <class F>
static void with_kernel(bool periodic, bool accurate, bool poly, bool close, F&& f) {
  const auto flag = [](bool v, auto&& g) { v ? g(std::true_type{}) : g(std::false_type{}); };
  flag(periodic, [&](auto p) {
    flag(close, [&](auto c) {
      if (accurate) f(p, std::integral_constant<int, K_ACC>{}, c);
      else if (poly) f(p, std::integral_constant<int, K_POLY>{}, c);
      else f(p, std::integral_constant<int, K_AS>{}, c);
    });
  });
}

// Targets per walk group: 32 fill a warp, but a small box then leaves most of
// the chip idle, and smaller groups share each target between lanes.  The
// largest power of two that still makes about 1,700 groups (of ~2,960 resident
// warps) was the fastest: walk ms at 32 / 16 / 8 / 4 / 2 / 1 targets for 4,096
// particles .173 .123 .108 .085 .073 .082; 8,000: .218 .160 .132 .110 .134
// .136; 13,824: .254 .181 .144 .173 .196 .244; 32,768: .356 .224 .255 .306
// .419 .574; 110,592: .452 .467 .601 .834 1.18 1.65.
int walk_group_size(int64_t n) {
  int size = WALK_TARGETS;
  while (size > 1 && n < (int64_t)size * 1700) size >>= 1;
  return size;
}

// (a handle may take several of the kernels, call by call)
int walk_blocks_per_sm(bool periodic, bool accurate) {
  int nb = 1;
  for (const bool poly : {false, true})
    for (const bool close : {false, true})
      with_kernel(periodic, accurate, poly, close, [&](auto p, auto k, auto c) {
        nb = std::max(nb, blocks_for<decltype(p)::value, decltype(k)::value, decltype(c)::value>());
      });
  return nb;
}

// Interpolation at the Chebyshev nodes of [0, x_max] of log2 of the A&S
// 7.1.26 erfc.  On x_max <= 3.6 (a cut of 5 r_s is x = 3.54) the polynomial stays
// within 2e-8 of that function, absolute, and its FP32 evaluation within 8e-8
// (the A&S form itself in FP32: 3.9e-7), so the walk takes one reciprocal less per
// pair; longer cuts keep the A&S form.
//
// Some pairs lie beyond the cut: monopoles by their half side, leaves of the
// aperiodic walk by that of their cell, all of them when the softening is long.
// Out there 2^P keeps falling to 0 for cuts from 3.65 r_s on, but for shorter ones
// P turns and rises without bound (at 2 r_s from 1.57 r_cut on).  `end` is the
// distance up to which its FP32 evaluation was found within 1e-7 of the function
// (at 65 points of the fit, then in steps of 1 %); beyond it the A&S form serves.
ErfcPoly erfc_poly(double x_max, double x_far) {
  ErfcPoly out{};
  if (!(x_max <= 3.6)) return out;
  const auto tail = [](double x) {  // the A&S form times exp(x^2)
    const double t = 1.0 / (1.0 + 0.3275911 * x);
    return t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))));
  };
  constexpr int N = POLY_DEGREE + 1;
  double node[N], div[N];
  for (int i = 0; i < N; ++i) {
    const double x = 0.5 * x_max * (1.0 - std::cos(M_PI * (i + 0.5) / N));
    node[i] = x;
    div[i] = std::log2(tail(x)) - x * x / std::log(2.0);
  }
  for (int k = 1; k < N; ++k)  // Newton's divided differences
    for (int i = N - 1; i >= k; --i) div[i] = (div[i] - div[i - 1]) / (node[i] - node[i - k]);
  double* c = out.coef;
  c[0] = div[N - 1];
  for (int k = N - 2; k >= 0; --k) {  // c <- c (x - node[k]) + div[k]
    for (int i = N - 1; i > 0; --i) c[i] = c[i - 1] - node[k] * c[i];
    c[0] = div[k] - node[k] * c[0];
  }
  const auto holds = [&](double x) {
    float p = (float)c[N - 1];
    for (int k = N - 2; k >= 0; --k) p = std::fma(p, (float)x, (float)c[k]);
    return std::fabs(std::exp2((double)p) - tail(x) * std::exp(-x * x)) <= 1e-7;  // (false for a NaN)
  };
  for (int i = 0; i <= 64; ++i)
    if (!holds(x_max * i / 64.0)) return out;
  out.end = x_max;
  for (double x = x_max; out.end < x_far && holds(x);) {
    out.end = x;
    x = std::min(1.01 * x, x_far);
    if (x == x_far && holds(x)) out.end = x;
  }
  return out;
}

size_t walk_stack_words(int grid) {
  return (size_t)grid * WALK_WARPS * STACK_ENTRIES * 4;  // one 16-byte entry = 4 words
}

void launch_walk(const WalkArgs& a, int grid, cudaStream_t s) {
  with_kernel(a.periodic != 0, a.accurate != 0, a.poly != 0, a.close != 0, [&](auto p, auto k, auto c) {
    launch_t<decltype(p)::value, decltype(k)::value, decltype(c)::value>(a, grid, s);
  });
  TPM_LAUNCH_CHECK();
}

// The count is on the device (zero in nearly every evaluation): one wave.
void launch_deferred(const WalkArgs& a, cudaStream_t s) {
  k_deferred<<<148, 64, 0, s>>>(a);
  TPM_LAUNCH_CHECK();
}

}  // namespace tpm
