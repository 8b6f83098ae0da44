// Intersection area and its adjoint.
//
// Forward: area(A_i ∩ B_i) = the shoelace sum over the boundary of A∩B, i.e.
// over the pieces of A's edges inside B and of B's edges inside A, found by
// the same slab / parity pass as the adjoint below (area mode).  Pairs whose
// crossings are not all clean, whose polygons do not fit the shared-memory
// staging, or whose area the crossing-rounding bound does not pin to 1e-10 are
// clipped by GPC instead (prt_overlay.cu, area-only mode: the clip result is
// reduced to its shoelace area in place and never written out).  The fast
// path assumes what GPC's output implies for map layers: the rings of a
// polygon do not cross each other or themselves, and hole rings are flagged.
//
// Backward: d area / d vertex by the boundary integral, recomputed from the
// input polygons rather than stored by the forward pass.  The boundary of
// A∩B is made of the pieces of A's edges inside B and of B's edges inside A
// (even-odd fill, GPC's parity rule).  For an edge p -> q traversed with the
// material on its left (ring orientation sign s: +1 for CCW outer rings and CW
// holes), outward normal N = s (q.y - p.y, p.x - q.x), and inside parameter
// intervals [t0, t1]:
//     d area / d q += N sum (t1^2 - t0^2) / 2
//     d area / d p += N sum ((t1 - t0) - (t1^2 - t0^2) / 2)
// One warp per pair: lanes take edges of A (then of B); each lane finds its
// edge's crossings with the other polygon, in increasing t, and classifies
// the intervals between them (by crossing parity along the ring, or by the
// even-odd test of each midpoint when a crossing is not clean; see
// pair_boundary).  Contributions are scaled by the upstream gradient and
// accumulated with atomicAdd, since a polygon may appear in many pairs.  Both
// directions run in stages: pairs of one-ring polygons of at most 8 vertices a
// thread each (area_tiny_kernel; with few pairs the next stage does them too),
// polygons of up to 64 vertices staged in shared memory (backward: pairs of 32
// together in a form of their own), the pairs that do not fit listed for a
// 128-vertex staging, then a 256-vertex one, and larger ones on a global-memory
// path (backward, on the 128-vertex stage) or the GPC clip (forward).
#include <cuda_runtime.h>

#include <atomic>
#include <climits>

#include "prt_internal.cuh"
#include "prt_overlay.cuh"

namespace prt {
namespace {

struct Poly {
  const int64_t *ring_vert;
  const int32_t *ring_hole;
  const double *xy;
  int64_t r0, r1;
};

__device__ inline bool inside_evenodd(const Poly &P, double px, double py) {
  bool c = false;
  for (int64_t r = P.r0; r < P.r1; r++) {
    const int64_t v0 = P.ring_vert[r], v1 = P.ring_vert[r + 1];
    const int64_t n = v1 - v0;
    for (int64_t i = 0; i < n; i++) {
      const int64_t j = (i + 1 == n) ? 0 : i + 1;
      const double ax = __ldg(&P.xy[2 * (v0 + i)]), ay = __ldg(&P.xy[2 * (v0 + i) + 1]);
      const double bx = __ldg(&P.xy[2 * (v0 + j)]), by = __ldg(&P.xy[2 * (v0 + j) + 1]);
      if ((ay > py) != (by > py)) {
        const double xi = ax + (py - ay) * (bx - ax) / (by - ay);
        if (px < xi) c = !c;
      }
    }
  }
  return c;
}

// smallest crossing parameter t of p + t r with the edges of P, t in (t_lo, 1)
__device__ inline double next_crossing(const Poly &P, double px, double py, double rx, double ry, double t_lo) {
  double best = 1.0;
  for (int64_t r = P.r0; r < P.r1; r++) {
    const int64_t v0 = P.ring_vert[r], v1 = P.ring_vert[r + 1];
    const int64_t n = v1 - v0;
    for (int64_t k = 0; k < n; k++) {
      const int64_t l = (k + 1 == n) ? 0 : k + 1;
      const double ax = __ldg(&P.xy[2 * (v0 + k)]), ay = __ldg(&P.xy[2 * (v0 + k) + 1]);
      const double sx = __ldg(&P.xy[2 * (v0 + l)]) - ax, sy = __ldg(&P.xy[2 * (v0 + l) + 1]) - ay;
      const double den = rx * sy - ry * sx;
      if (den == 0.0) continue;
      const double apx = ax - px, apy = ay - py;
      const double t = (apx * sy - apy * sx) / den;
      const double u = (apx * ry - apy * rx) / den;
      if (t > 0.0 && t < 1.0 && u >= 0.0 && u <= 1.0 && t > t_lo && t < best) best = t;
    }
  }
  return best;
}

// Pieces of A's boundary inside B, for the edges handled by this lane.
__device__ void pieces(const Poly &A, const Poly &B, double w, double *grad, int lane) {
  for (int64_t r = A.r0; r < A.r1; r++) {
    const int64_t v0 = A.ring_vert[r], v1 = A.ring_vert[r + 1];
    const int64_t n = v1 - v0;
    if (n < 2) continue;
    // ring orientation (warp-cooperative shoelace)
    double sa = 0.0;
    for (int64_t i = lane; i < n; i += 32) {
      const int64_t j = (i + 1 == n) ? 0 : i + 1;
      sa += A.xy[2 * (v0 + i)] * A.xy[2 * (v0 + j) + 1] - A.xy[2 * (v0 + j)] * A.xy[2 * (v0 + i) + 1];
    }
    for (int o = 16; o; o >>= 1) sa += __shfl_xor_sync(0xffffffffu, sa, o);
    // material on the left: CCW outer rings and CW hole rings (s = +1)
    const bool hole = A.ring_hole && A.ring_hole[r];
    const double s = (sa >= 0.0 ? 1.0 : -1.0) * (hole ? -1.0 : 1.0);
    for (int64_t i = lane; i < n; i += 32) {
      const int64_t j = (i + 1 == n) ? 0 : i + 1;
      const double px = A.xy[2 * (v0 + i)], py = A.xy[2 * (v0 + i) + 1];
      const double qx = A.xy[2 * (v0 + j)], qy = A.xy[2 * (v0 + j) + 1];
      const double rx = qx - px, ry = qy - py;
      double it = 0.0, i1 = 0.0;
      double t0 = 0.0;
      for (;;) {
        const double t1 = next_crossing(B, px, py, rx, ry, t0);
        const double tm = 0.5 * (t0 + t1);
        if (t1 > t0 && inside_evenodd(B, px + tm * rx, py + tm * ry)) {
          const double a = 0.5 * (t1 * t1 - t0 * t0);
          it += a;
          i1 += (t1 - t0) - a;
        }
        if (t1 >= 1.0) break;
        t0 = t1;
      }
      if (it != 0.0 || i1 != 0.0) {
        const double nx = w * s * ry, ny = -w * s * rx;
        atomicAdd(&grad[2 * (v0 + j)], nx * it);
        atomicAdd(&grad[2 * (v0 + j) + 1], ny * it);
        atomicAdd(&grad[2 * (v0 + i)], nx * i1);
        atomicAdd(&grad[2 * (v0 + i) + 1], ny * i1);
      }
    }
  }
}

// ---- shared-memory adjoint (pairs up to kBwdLargeV vertices per polygon) ----
// The same boundary pieces with both polygons staged in shared memory, and
// the candidate edges of the other polygon found through y slabs instead of
// a scan over all of its edges.  The pair's common y range (float, rounded
// outwards) is cut into kSlabs slabs; slab s of polygon Q holds a bitmask of
// Q's edges whose float box reaches slab s (built by a warp bit transpose of
// each edge's slab range).  The slab index is a monotone function of the
// float y, so two y ranges that overlap always share a slab and the masks
// never drop a candidate:
//   crossings of an edge: the OR of the slab masks over its y range, then the
//     float box test and the exact FP64 crossing expression of
//     next_crossing, so the crossing set equals the exhaustive scan's;
//   midpoint of an interval: only edges whose y range holds the midpoint's y
//     can straddle it, and they all sit in the midpoint's slab; the even-odd
//     test is inside_evenodd's expression.
// Each lane takes one edge (the edges of A and of B in one pass); the
// crossing parameters are sorted and deduplicated, which gives the intervals
// of next_crossing's repeated minimum search.  The two gradient contributions
// a vertex receives (as the end of one edge, as the start of the next) are
// summed across neighbouring lanes before the atomics.  Edges with more than
// kBwdMaxT crossings take the global-memory path (next_crossing).
constexpr int kBwdOneV = 32;  // both polygons' vertices together (gradients only)
constexpr int kBwdSmallV = 64;
constexpr int kBwdMidV = 128;
constexpr int kBwdLargeV = 256;  // BwdPoly's 8-bit vertex indices hold no more
constexpr int kBwdMaxT = 16;
// Warps (pairs) per block of the V-vertex stage: the 256-vertex staging takes 23 KB a
// pair, 8 pairs an SM.
constexpr int bwd_warps(int V) { return V > kBwdMidV ? 2 : 4; }
constexpr int kSlabs = 32;
constexpr unsigned kFullMask = 0xffffffffu;

template <int V>
struct BwdPoly {  // one polygon in shared memory (up to V vertices)
  float4 bb[V];                    // edge k's box (x_lo, y_lo, x_hi, y_hi), rounded outwards
  double x[V], y[V];
  int16_t ringv[33];                      // first vertex of ring r; ringv[rings] = the vertex count
  int8_t sgn[V];                   // orientation sign of edge k (0: ring of < 2 vertices)
  uint8_t nxt[V];                  // end vertex of edge k
  uint8_t rst[V];                  // first vertex of edge k's ring
};

// Slab masks of one polygon's edges.
template <int V>
struct BwdSlabs {
  uint32_t y[V / 32][kSlabs];  // word c of slab s, bit k = edge 32 c + k reaches slab s
  uint32_t x[V / 32][kSlabs];
};

// Crossings of a pair, chained by the edge of the searched polygon.
constexpr int bwd_crossings(int V) { return V > kBwdMidV ? 192 : 128; }
template <int V>
struct BwdCrossings {
  double u[bwd_crossings(V)];       // parameter on that edge, negative where the edge leaves the other polygon
  uint16_t next[bwd_crossings(V)];  // 1 + the next crossing of the same edge (0: none)
  uint32_t head[V];                 // 1 + the edge's first crossing (0: none)
  uint32_t count;                   // crossings found (beyond the room too)
};

template <int V>
struct BwdPair {  // one warp's shared memory
  BwdPoly<V> poly[2];
  BwdSlabs<V> slab;  // of the polygon that is searched
  BwdCrossings<V> cross;
};

// coordinate -> slab: monotone non-decreasing (round-to-nearest float steps
// and a clamp), which is what makes the slab masks conservative.
struct SlabGrid {
  float v0, scale;
  __device__ int operator()(float v) const {
    const float f = __fmul_rn(__fsub_rn(v, v0), scale);
    return (int)fminf(fmaxf(f, 0.0f), (float)(kSlabs - 1));
  }
};

__device__ inline SlabGrid slab_grid(float lo, float hi) {
  const float span = __fsub_rn(hi, lo);
  return SlabGrid{lo, span > 1e-30f ? __fdiv_rn((float)kSlabs, span) : 0.0f};
}

// Smallest value of the warp, by one integer reduction of the order-preserving
// image.
__device__ __forceinline__ float warp_fmin(float v) {
  const int i = __float_as_int(v);
  const int k = __reduce_min_sync(kFullMask, i >= 0 ? i : i ^ 0x7fffffff);
  return __int_as_float(k >= 0 ? k : k ^ 0x7fffffff);
}

// Stages both polygons of a pair (A from rings [ra0, ra1) of LA, B from
// [rb0, rb1) of LB) with their ring links, orientation signs and edge boxes;
// the loads of the two are issued together.  nv[p] is polygon p's vertex
// count, vb[p] its first vertex, ext[p] the float extent of its edge boxes.
// Returns false (nothing staged) when a polygon has more than V
// vertices or more than 31 rings.
template <int V>
__device__ inline bool bwd_load_pair(const LayerDev &LA, int64_t ra0, int64_t ra1, const LayerDev &LB, int64_t rb0,
                                     int64_t rb1, BwdPoly<V> *M, int *nv, int64_t *vb, float4 *ext) {
  const int lane = threadIdx.x & 31;
  const int nr[2] = {(int)(ra1 - ra0), (int)(rb1 - rb0)};
  nv[0] = nv[1] = INT_MAX;
  if (nr[0] > 31 || nr[1] > 31) return false;
  int64_t rv[2] = {0, 0};
  int hl[2] = {0, 0};
  if (lane <= nr[0]) rv[0] = LA.ring_vert[ra0 + lane];
  if (lane <= nr[1]) rv[1] = LB.ring_vert[rb0 + lane];
  if (lane < nr[0] && LA.ring_hole) hl[0] = LA.ring_hole[ra0 + lane];
  if (lane < nr[1] && LB.ring_hole) hl[1] = LB.ring_hole[rb0 + lane];
#pragma unroll
  for (int p = 0; p < 2; p++) {
    vb[p] = __shfl_sync(kFullMask, rv[p], 0);
    nv[p] = (int)(__shfl_sync(kFullMask, rv[p], nr[p]) - vb[p]);
  }
  if (nv[0] > V || nv[1] > V) return false;
#pragma unroll
  for (int p = 0; p < 2; p++)
    if (lane <= nr[p]) M[p].ringv[lane] = (int16_t)(rv[p] - vb[p]);
  __syncwarp();
  const float inf = __int_as_float(0x7f800000);
  float4 e[2] = {make_float4(inf, inf, -inf, -inf), make_float4(inf, inf, -inf, -inf)};
  double term[2][V / 32];  // shoelace terms of this lane's vertices
  int rix[2][V / 32];      // and their rings
#pragma unroll
  for (int t = 0; t < V / 32; t++) {
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const LayerDev &L = p ? LB : LA;
      BwdPoly<V> &Q = M[p];
      const int i = 32 * t + lane;
      term[p][t] = 0.0;
      rix[p][t] = -1;
      if (i < nv[p]) {
        int r = 0;
        while (Q.ringv[r + 1] <= i) r++;
        const int v0 = Q.ringv[r], j = i + 1 == Q.ringv[r + 1] ? v0 : i + 1;
        const double xi = L.xy[2 * (vb[p] + i)], yi = L.xy[2 * (vb[p] + i) + 1];
        const double xj = L.xy[2 * (vb[p] + j)], yj = L.xy[2 * (vb[p] + j) + 1];
        term[p][t] = xi * yj - xj * yi;
        rix[p][t] = r;
        Q.x[i] = xi;
        Q.y[i] = yi;
        Q.nxt[i] = (uint8_t)j;
        Q.rst[i] = (uint8_t)v0;
        const float4 b = make_float4(__double2float_rd(fmin(xi, xj)), __double2float_rd(fmin(yi, yj)),
                                     __double2float_ru(fmax(xi, xj)), __double2float_ru(fmax(yi, yj)));
        Q.bb[i] = b;
        e[p] = make_float4(fminf(e[p].x, b.x), fminf(e[p].y, b.y), fmaxf(e[p].z, b.z), fmaxf(e[p].w, b.w));
      }
    }
  }
  // ring orientations: material on the left for CCW outer rings and CW holes
#pragma unroll
  for (int p = 0; p < 2; p++) {
    for (int r = 0; r < nr[p]; r++) {
      double sa = 0.0;
#pragma unroll
      for (int t = 0; t < V / 32; t++) sa += rix[p][t] == r ? term[p][t] : 0.0;
      for (int o = 16; o; o >>= 1) sa += __shfl_xor_sync(kFullMask, sa, o);
      const bool hole = __shfl_sync(kFullMask, hl[p], r) != 0;
      const int n = M[p].ringv[r + 1] - M[p].ringv[r];
      const int8_t sg = n < 2 ? 0 : (int8_t)((sa >= 0.0 ? 1 : -1) * (hole ? -1 : 1));
#pragma unroll
      for (int t = 0; t < V / 32; t++)
        if (rix[p][t] == r) M[p].sgn[32 * t + lane] = sg;
    }
    ext[p] = make_float4(warp_fmin(e[p].x), warp_fmin(e[p].y), -warp_fmin(-e[p].z), -warp_fmin(-e[p].w));
  }
  __syncwarp();
  return true;
}

// 32 x 32 bit matrix transpose across the warp: bit i of lane l's result is
// bit l of lane i's input (recursive exchange of off-diagonal blocks).
__device__ inline uint32_t bit_transpose(uint32_t x) {
  const int lane = threadIdx.x & 31;
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j; j >>= 1, m ^= m << j) {
    const uint32_t t = __shfl_xor_sync(kFullMask, x, j);
    x = (lane & j) ? ((x & ~m) | ((t >> j) & m)) : ((x & m) | ((t << j) & ~m));
  }
  return x;
}

// y and x slab masks of two staged polygons of up to 32 edges each (four
// independent transposes).
template <int V>
__device__ inline void bwd_slabs_both(const BwdPoly<V> *M, int na, int nb, const SlabGrid &gy, const SlabGrid &gx,
                                      BwdSlabs<V> &SA, BwdSlabs<V> &SB) {
  const int lane = threadIdx.x & 31;
  uint32_t ry[2] = {0, 0}, rx[2] = {0, 0};
#pragma unroll
  for (int p = 0; p < 2; p++)
    if (lane < (p ? nb : na)) {
      const float4 b = M[p].bb[lane];
      ry[p] = (kFullMask >> (31 - gy(b.w))) & (kFullMask << gy(b.y));
      rx[p] = (kFullMask >> (31 - gx(b.z))) & (kFullMask << gx(b.x));
    }
  SA.y[0][lane] = bit_transpose(ry[0]);
  SA.x[0][lane] = bit_transpose(rx[0]);
  SB.y[0][lane] = bit_transpose(ry[1]);
  SB.x[0][lane] = bit_transpose(rx[1]);
  __syncwarp();
}

// y and x slab masks of a staged polygon (two independent transposes per word).
template <int V>
__device__ inline void bwd_slabs(const BwdPoly<V> &Q, int nq, const SlabGrid &gy, const SlabGrid &gx, BwdSlabs<V> &S) {
  const int lane = threadIdx.x & 31;
  for (int c = 0; 32 * c < nq; c++) {
    const int k = 32 * c + lane;
    uint32_t ry = 0, rx = 0;
    if (k < nq) {
      const float4 b = Q.bb[k];
      ry = (kFullMask >> (31 - gy(b.w))) & (kFullMask << gy(b.y));
      rx = (kFullMask >> (31 - gx(b.z))) & (kFullMask << gx(b.x));
    }
    S.y[c][lane] = bit_transpose(ry);
    S.x[c][lane] = bit_transpose(rx);
  }
  __syncwarp();
}

// One edge whose crossings overflow the per-lane list: the global-memory path.
__device__ __noinline__ void bwd_edge_global(const Poly &Qg, double px, double py, double rx, double ry, double *it,
                                             double *i1) {
  double t0 = 0.0;
  for (;;) {
    const double t1 = next_crossing(Qg, px, py, rx, ry, t0);
    const double tm = 0.5 * (t0 + t1);
    if (t1 > t0 && inside_evenodd(Qg, px + tm * rx, py + tm * ry)) {
      const double a = 0.5 * (t1 * t1 - t0 * t0);
      *it += a;
      *i1 += (t1 - t0) - a;
    }
    if (t1 >= 1.0) break;
    t0 = t1;
  }
}

// Even-odd test of (mx, my) against staged polygon Q through the slab of
// my: inside_evenodd's expression over the edges that can straddle my.
template <int V>
__device__ inline bool bwd_inside(const BwdPoly<V> &Q, const BwdSlabs<V> &S, int nwq, const float4 &qe,
                                  const SlabGrid &g, double mx, double my) {
  const float fy = __double2float_rn(my);
  if (fy < qe.y || fy > qe.w) return false;  // no edge of Q straddles my
  const int s = g(fy);
  bool in = false;
  for (int c = 0; c < nwq; c++) {
    uint32_t bits = S.y[c][s];
    while (bits) {
      const int k = 32 * c + __ffs(bits) - 1;
      bits &= bits - 1;
      const int l = Q.nxt[k];
      const double ay = Q.y[k], by = Q.y[l];
      if ((ay > my) != (by > my)) {
        const double ax = Q.x[k], bx = Q.x[l];
        const double xi = ax + (my - ay) * (bx - ax) / (by - ay);
        if (mx < xi) in = !in;
      }
    }
  }
  return in;
}

// Candidate edges of Q (mask word c) for an edge whose box covers y slabs
// [s0, s1] and x slabs [x0, x1].
template <int V>
__device__ inline uint32_t bwd_cands(const BwdSlabs<V> &S, int c, int s0, int s1, int x0, int x1) {
  uint32_t ybits = 0, xbits = 0;
  for (int s = s0; s <= s1; s++) ybits |= S.y[c][s];
  for (int s = x0; s <= x1; s++) xbits |= S.x[c][s];
  return ybits & xbits;
}

// One edge p -> p + r against staged polygon Q by the definition: every
// crossing by next_crossing's test (kBwdMaxT at most, else the global-memory
// path), sorted and deduplicated, and every interval by its midpoint.
template <int V>
__device__ __noinline__ void bwd_edge_exact(const BwdPoly<V> &Q, const BwdSlabs<V> &S, int nwq, const float4 &qe, const SlabGrid &g,
                                            const SlabGrid &gx, const float4 &pb, double px, double py, double rx,
                                            double ry, const Poly &Qg, double *it_out, double *i1_out) {
  double ts[kBwdMaxT];
  int nt = 0;
  bool over = false;
  const int s0 = g(pb.y), s1 = g(pb.w), x0 = gx(pb.x), x1 = gx(pb.z);
  for (int c = 0; c < nwq; c++) {
    uint32_t bits = bwd_cands(S, c, s0, s1, x0, x1);
    while (bits) {
      const int k = 32 * c + __ffs(bits) - 1;
      bits &= bits - 1;
      const float4 b = Q.bb[k];
      if (b.w < pb.y || b.y > pb.w || b.z < pb.x || b.x > pb.z) continue;
      const int l = Q.nxt[k];
      const double ax = Q.x[k], ay = Q.y[k], bx = Q.x[l], by = Q.y[l];
      const double sx = bx - ax, sy = by - ay;
      const double den = rx * sy - ry * sx;
      if (den == 0.0) continue;
      const double apx = ax - px, apy = ay - py;
      const double t = (apx * sy - apy * sx) / den;
      const double u = (apx * ry - apy * rx) / den;
      if (t > 0.0 && t < 1.0 && u >= 0.0 && u <= 1.0) {
        if (nt < kBwdMaxT) ts[nt++] = t;
        else over = true;
      }
    }
  }
  double it = 0.0, i1 = 0.0;
  if (over) {
    bwd_edge_global(Qg, px, py, rx, ry, &it, &i1);
  } else {
    for (int a = 1; a < nt; a++) {  // sort, then drop duplicates
      const double v = ts[a];
      int b = a - 1;
      while (b >= 0 && ts[b] > v) {
        ts[b + 1] = ts[b];
        b--;
      }
      ts[b + 1] = v;
    }
    int m = 0;
    for (int a = 0; a < nt; a++)
      if (m == 0 || ts[a] > ts[m - 1]) ts[m++] = ts[a];
    for (int a = 0; a <= m; a++) {
      const double t0 = a == 0 ? 0.0 : ts[a - 1], t1 = a < m ? ts[a] : 1.0;
      const double tm = 0.5 * (t0 + t1);
      if (bwd_inside(Q, S, nwq, qe, g, px + tm * rx, py + tm * ry)) {
        const double aa = 0.5 * (t1 * t1 - t0 * t0);
        it += aa;
        i1 += (t1 - t0) - aa;
      }
    }
  }
  *it_out = it;
  *i1_out = i1;
}

// pieces() for both polygons of a staged pair, in rounds of 32 edges (one per
// lane): first the edges of the polygon with fewer, P, which search the other,
// Q, for crossings; then Q's edges, which find theirs in chains that the
// search left: a crossing of p + t r and a + u s has t = tn / den and u = un /
// den from the same three products, whichever edge looks, so each is computed
// once.  ext[0], ext[1]: the float extents of A and B.
//
// What is inside: by the midpoint of every interval between crossings (the
// definition, bwd_edge_exact), or, while the pair's crossings are all clean,
// from the crossings alone: the state at an edge's start (the ring's first
// edge by the midpoint of a piece of it, later ones flip with the number of
// crossings before them on the ring: a prefix XOR carried between rounds) and
// one signed term per crossing, +1 where the edge enters the other polygon
// and -1 where it leaves it, by the side of the other edge that its ring's
// orientation sign says is inside.  With the state s1 at the edge's end,
//     sum (t1 - t0)         = s1 - sum sign t
//     sum (t1^2 - t0^2) / 2 = (s1 - sum sign t^2) / 2
// so no list of crossings is kept, sorted or bounded.  A crossing is clean
// when it is well inside both edges (t and u at least 1e-9 from 0 and 1) and
// the edges are not nearly parallel; collinear overlapping edges are not
// clean, nor is an edge whose signed crossings do not add up to its change of
// state (rings that cross, hole rings that are not flagged).  From the first
// round with an unclean edge on, the pair goes by the definition.
// (With a sorted register list per edge, of 4 crossings in gradient mode and 6
// in area mode, 1M pairs of 16-64-vertex stars took 6.89 ms backward and 6.11
// forward against 6.47 and 5.63 with the sums; of 50k pairs of 4-160 vertices,
// whose long edges run along the other's spikes, 2.2 and 1.16 ms and a longer
// GPC list against 1.09 and 1.05.)

// Area mode of the same pass (the forward): per edge, the inside length
// L = sum (t1 - t0) over its inside intervals contributes
//     s * L * cross(p - O, q - p) / 2
// to area(A∩B) (the shoelace term of each inside piece, about a pair-local
// origin O), and every clean crossing adds a bound on how far GPC's own
// vertex can lie from it: a vertex error of ~eps * max|coordinate| /
// sin(angle) times the two edges' lengths,
//     (|r|_1 + |s|_1) * |r|_1 * |s|_1 / |r x s|  (times eps * max|coordinate|).
struct AreaSum {
  double area;  // twice the area, summed over the warp by the caller
  double err;   // the crossing error bound above, without its eps * max|coordinate| factor
};

// Returns false in area mode as soon as any crossing of the pair is unclean
// (the caller then clips the pair with GPC); in gradient mode it always runs
// to the end, by the definition from the first unclean crossing on.
// kOne (na + nb <= kBwdOneV): both polygons' edges in one round, every edge searching for
// itself: two half-empty rounds and the chains cost more than finding each crossing
// twice.
template <bool kArea, bool kOne, int V>
__device__ inline bool pair_boundary(BwdPair<V> &W, const float4 *ext, int na, int nb, const SlabGrid &g,
                                     const SlabGrid &gx, double w, double *ga, double *gb, int64_t va, int64_t vb,
                                     const Poly &Ag, const Poly &Bg, double ox, double oy, AreaSum *acc) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  BwdCrossings<V> &X = W.cross;
  const int searcher = nb < na ? 1 : 0;
  int masks = 1 - searcher;  // the polygon W.slab belongs to
  static_assert(!kOne || sizeof(BwdSlabs<V>) <= sizeof(BwdCrossings<V>), "A's masks in the place of the chains");
  BwdSlabs<V> &SA = *reinterpret_cast<BwdSlabs<V> *>(&X);
  if constexpr (kOne) {
    bwd_slabs_both(W.poly, na, nb, g, gx, SA, W.slab);
  } else {
    bwd_slabs(W.poly[masks], masks ? nb : na, g, gx, W.slab);
    for (int k = lane; k < (masks ? nb : na); k += 32) X.head[k] = 0;
    if (lane == 0) X.count = 0;
    __syncwarp();
  }
  bool exact = false;  // by the definition from here on (sticky)
  double area2 = 0.0, err = 0.0;
  for (int half = 0; half < (kOne ? 1 : 2); half++) {
    // kOne: lanes [0, na) have A's edges, [na, na + nb) B's
    const int side = kOne ? (lane < na ? 0 : 1) : half ? 1 - searcher : searcher;
    const int lane0 = kOne && side ? na : 0;
    const BwdPoly<V> &P = W.poly[side], &Q = W.poly[1 - side];
    const int np = side ? nb : na, nq = side ? na : nb;
    const int nwq = (nq + 31) >> 5;
    bool carry = false;  // inside state after the last edge of the previous round
    for (int e0 = 0; e0 < (kOne ? 1 : np); e0 += 32) {
      const int i = e0 + lane - lane0;
      const bool valid = i < np && P.sgn[i] != 0;
      const int j = valid ? P.nxt[i] : 0;
      double px = 0.0, py = 0.0, qx = 0.0, qy = 0.0;
      float4 pb = make_float4(0.f, 0.f, 0.f, 0.f);
      if (valid) {
        px = P.x[i];
        py = P.y[i];
        qx = P.x[j];
        qy = P.y[j];
        pb = P.bb[i];
      }
      const double rx = qx - px, ry = qy - py;
      double c1 = 0.0, c2 = 0.0;  // sums of sign t and sign t^2 over the edge's clean crossings
      int c0 = 0;                 // and of the signs
      int m = 0;                  // their number
      double tfirst = 1.0;        // the first one
      if (half == 0 && !exact) {
        bool unclean = false;
        if (valid) {
          const bool material_left = P.sgn[i] > 0;
          const double rl = fabs(rx) + fabs(ry);
          const int s0 = g(pb.y), s1 = g(pb.w), x0 = gx(pb.x), x1 = gx(pb.z);
          for (int c = 0; c < (kOne ? 1 : nwq); c++) {
            uint32_t bits = bwd_cands(kOne && side ? SA : W.slab, c, s0, s1, x0, x1);
            while (bits) {
              const int k = 32 * c + __ffs(bits) - 1;
              bits &= bits - 1;
              const float4 b = Q.bb[k];
              if (b.w < pb.y || b.y > pb.w || b.z < pb.x || b.x > pb.z) continue;
              const int l = Q.nxt[k];
              const double ax = Q.x[k], ay = Q.y[k], bx = Q.x[l], by = Q.y[l];
              const double sx = bx - ax, sy = by - ay;
              const double den = rx * sy - ry * sx;
              const double apx = ax - px, apy = ay - py;
              const double tn = apx * sy - apy * sx;
              const double un = apx * ry - apy * rx;
              if (den == 0.0) {
                unclean |= tn == 0.0 || un == 0.0;  // collinear
                continue;
              }
              // t = tn / den and u = un / den, with the signs of den folded in
              const double d = fabs(den), tol = 1e-9 * d;
              const double tt = den > 0.0 ? tn : -tn, uu = den > 0.0 ? un : -un;
              if (tt < -tol || tt > d + tol || uu < -tol || uu > d + tol) continue;  // next_crossing rejects it
              const double sl = fabs(sx) + fabs(sy);
              if (!(tt > tol && tt < d - tol && uu > tol && uu < d - tol && d > 1e-6 * rl * sl)) {
                unclean = true;
                continue;
              }
              // seen from both edges
              if constexpr (kArea) err += (kOne ? 1.0 : 2.0) * ((rl + sl) * rl * sl / d);
              const double t = tn / den;  // next_crossing's t
              // den > 0: P's edge goes from the left of Q's edge to its right,
              // out of Q where Q's material is on the left, and Q's edge the
              // other way
              const bool leaves = (den > 0.0) == (Q.sgn[k] > 0);
              const double st = leaves ? -t : t;
              c0 += leaves ? -1 : 1;
              c1 += st;
              c2 += st * t;
              tfirst = fmin(tfirst, t);
              m++;
              if constexpr (!kOne) {
                const double u = un / den;  // and seen from the other edge
                const uint32_t x = atomicAdd(&X.count, 1u);
                if (x < (uint32_t)bwd_crossings(V)) {
                  X.u[x] = (den < 0.0) == material_left ? -u : u;
                  X.next[x] = (uint16_t)atomicExch(&X.head[k], x + 1);
                } else {
                  unclean = true;
                }
              }
            }
          }
        }
        exact = __any_sync(kFullMask, unclean);
        if constexpr (kArea) {
          if (exact) return false;
        }
      } else if (half == 1 && !exact && valid) {
        for (uint32_t x = X.head[i]; x;) {
          const double st = X.u[x - 1], t = fabs(st);
          c0 += st < 0.0 ? -1 : 1;
          c1 += st;
          c2 += st * t;
          tfirst = fmin(tfirst, t);
          m++;
          x = X.next[x - 1];
        }
      }
      double it = 0.0, i1 = 0.0;
      if (!exact) {
        const int rs = valid ? P.rst[i] : i;  // this edge's ring starts at edge rs
        // the first interval of each ring starting in this round, by its
        // midpoint: the whole warp tests it against all edges of the other polygon
        const bool rstart = valid && rs == i;
        const int rlane = rs + lane0;
        double mx0 = 0.0, my0 = 0.0;
        if (rstart) {
          const double tm = 0.5 * tfirst;
          mx0 = px + tm * rx;
          my0 = py + tm * ry;
        }
        bool first = false;
        for (unsigned q = __ballot_sync(kFullMask, rstart); q; q &= q - 1) {
          const int L = __ffs(q) - 1;
          const double mxl = __shfl_sync(kFullMask, mx0, L), myl = __shfl_sync(kFullMask, my0, L);
          bool in = false;
          const int sl = kOne ? (L < na ? 0 : 1) : side;
          const BwdPoly<V> &QL = W.poly[1 - sl];
          for (int k = lane; k < (sl ? na : nb); k += 32) {
            const int l = QL.nxt[k];
            const double ay = QL.y[k], by = QL.y[l];
            if ((ay > myl) != (by > myl)) {
              const double ax = QL.x[k], bx = QL.x[l];
              const double xi = ax + (myl - ay) * (bx - ax) / (by - ay);
              if (mxl < xi) in = !in;
            }
          }
          const bool inside = (__popc(__ballot_sync(kFullMask, in)) & 1) != 0;
          if (lane == L) first = inside;
        }
        const unsigned odd = __ballot_sync(kFullMask, (m & 1) != 0);
        const int from = rlane > e0 ? rlane - e0 : 0;
        const int par = __popc(odd & lt & ~((1u << from) - 1u)) & 1;
        const bool sf = __shfl_sync(kFullMask, first, from);
        const bool st = (rs >= e0 ? sf : carry) != (par != 0);  // inside state at the edge's start
        const bool end = st != ((m & 1) != 0);
        carry = __shfl_sync(kFullMask, end, 31);
        if (__any_sync(kFullMask, valid && (int)st + c0 != (int)end)) {
          exact = true;
          if constexpr (kArea) return false;
        }
        if (valid) {
          const double s1 = end ? 1.0 : 0.0;
          it = 0.5 * (s1 - c2);
          i1 = (s1 - c1) - it;
        }
      }
      if constexpr (!kArea) {
        if (exact) {
          if (!kOne && masks != 1 - side) {
            masks = 1 - side;
            __syncwarp();
            bwd_slabs(Q, nq, g, gx, W.slab);
          }
          if (valid)
            bwd_edge_exact(Q, kOne && side ? SA : W.slab, nwq, side ? ext[0] : ext[1], g, gx, pb, px, py, rx, ry,
                           side ? Ag : Bg, &it, &i1);
        }
      }
      if constexpr (kArea) {
        // it + i1 = sum (t1 - t0) over the inside intervals
        if (valid) area2 += P.sgn[i] * (it + i1) * ((px - ox) * ry - (py - oy) * rx);
        continue;
      }
      // contributions: it to the end vertex j, i1 to the start vertex i; the
      // lane of the next edge of the ring hands its start contribution over so
      // the shared vertex takes one atomic per coordinate
      double gxj = 0.0, gyj = 0.0, gxi = 0.0, gyi = 0.0;
      if (valid) {
        const double s = P.sgn[i];
        const double nx = w * s * ry, ny = -w * s * rx;
        gxj = nx * it;
        gyj = ny * it;
        gxi = nx * i1;
        gyi = ny * i1;
      }
      const int key = valid ? side << 8 | i : -1;             // this edge's start vertex
      const int kend = valid ? side << 8 | j : -2;            // its end vertex
      const int knext = __shfl_down_sync(kFullMask, key, 1);  // start vertex of the next lane's edge
      const int kprev = __shfl_up_sync(kFullMask, kend, 1);   // end vertex of the previous lane's edge
      const double hx = __shfl_down_sync(kFullMask, gxi, 1), hy = __shfl_down_sync(kFullMask, gyi, 1);
      const bool take = lane < 31 && knext == kend;  // the next lane's i1 part goes with mine
      const bool given = lane > 0 && kprev == key;   // mine went to the previous lane
      if (take) {
        gxj += hx;
        gyj += hy;
      }
      double *gr = side ? gb : ga;
      const int64_t vbase = side ? vb : va;
      if (valid && (gxj != 0.0 || gyj != 0.0)) {
        atomicAdd(&gr[2 * (vbase + j)], gxj);
        atomicAdd(&gr[2 * (vbase + j) + 1], gyj);
      }
      if (valid && !given && (gxi != 0.0 || gyi != 0.0)) {
        atomicAdd(&gr[2 * (vbase + i)], gxi);
        atomicAdd(&gr[2 * (vbase + i) + 1], gyi);
      }
    }
    __syncwarp();  // the crossings of the first half, for the second
  }
  if constexpr (kArea) {
    acc->area = area2;
    acc->err = err;
  }
  return true;
}

// Pairs with a polygon above V vertices: the global-memory path.
__device__ __noinline__ void bwd_pair_global(const Poly &A, const Poly &B, double w, double *ga, double *gb) {
  const int lane = threadIdx.x & 31;
  pieces(A, B, w, ga, lane);
  pieces(B, A, w, gb, lane);
}

// Pair lists of the staged launches: the first stage (V = kBwdSmallV) takes
// every pair and lists those with a polygon above V vertices (or 31 rings) in
// `defer`; the next stages (V = kBwdMidV, kBwdLargeV) take only the pairs the
// one before listed (`sel`, *sel_count of them).  The gradients of pairs too large for
// the last stage are taken on the global-memory path by the one before it, which has 16
// warps per SM for its 8 (10k pairs of 257-400 vertices: 28.5 ms against 40.9).
struct PairList {
  const int32_t *sel;                   // items of this launch (nullptr: pairs 0 .. n-1)
  const unsigned long long *sel_count;  // how many (device)
  int32_t *defer;                       // pairs this stage cannot stage (nullptr: none deferred)
  unsigned long long *defer_count;
};

__device__ __forceinline__ int64_t list_items(const PairList &L, int64_t n) {
  return L.sel ? (int64_t)min((unsigned long long)n, *L.sel_count) : n;
}

// 4 blocks of 4 warps per SM (up to 128 registers, no spills; measured at 1M
// pairs of 16-64-vertex stars, 5 blocks of the V = 64 kernel spill and run
// 10% slower).  The 256-vertex stage is bound by its shared memory: 4 blocks
// of 2 warps.  Before it, 50k pairs of 4-160 vertices (a third of them above
// 128) took 10.8 ms here on the global-memory path and 11.5 ms in the
// forward's GPC clip.
// The smallest stage is launched beside the 64-vertex one, in whose tail it runs:
// both take what area_tiny_kernel lists.
// kMixed: pairs of few vertices are taken here too, in one round.
template <int V, bool kMixed>
__global__ void __launch_bounds__(32 * bwd_warps(V), V > kBwdMidV ? 5 : 4) area_bwd_kernel(
    const int32_t *__restrict__ pa, const int32_t *__restrict__ pb, int64_t n, LayerDev base, LayerDev over,
    const double *__restrict__ upstream, double *grad_base, double *grad_over, PairList PL) {
  __shared__ BwdPair<V> sm[bwd_warps(V)];
  BwdPair<V> &W = sm[threadIdx.x >> 5];
  BwdPoly<V> *M = W.poly;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  if constexpr (V != kBwdOneV) cudaGridDependencySynchronize();
  if constexpr (V == kBwdSmallV) cudaTriggerProgrammaticLaunchCompletion();
  const int64_t items = list_items(PL, n);
  // a pair's ids are read one pair ahead and its ring ranges half a pair
  // ahead, so the staging of a pair waits only for its ring starts and
  // vertices
  auto ids = [&](int64_t k, int64_t *i, int64_t *a, int64_t *b) {
    *i = -1;
    *a = -1;
    *b = -1;
    if (k < items) {
      const int64_t j = PL.sel ? PL.sel[k] : k;
      if (j >= 0 && j < n) {
        const int64_t x = pa[j], y = pb[j];
        if (x >= 0 && x < base.n_poly && y >= 0 && y < over.n_poly) {
          *i = j;
          *a = x;
          *b = y;
        }
      }
    }
  };
  auto rings = [&](int64_t a, int64_t b, int64_t *r) {
    r[0] = r[1] = r[2] = r[3] = 0;
    if (a >= 0) {
      r[0] = base.poly_ring[a];
      r[1] = base.poly_ring[a + 1];
      r[2] = over.poly_ring[b];
      r[3] = over.poly_ring[b + 1];
    }
  };
  int64_t i, a, b, rr[4];
  ids(warp, &i, &a, &b);
  rings(a, b, rr);
  for (int64_t k = warp; k < items; k += nw) {
    int64_t in, an, bn, rn[4];
    ids(k + nw, &in, &an, &bn);
    bool fetched = false;
    if (a >= 0) {
      int nv[2];
      int64_t vb[2];
      float4 ext[2];
      const bool staged = bwd_load_pair(base, rr[0], rr[1], over, rr[2], rr[3], M, nv, vb, ext);
      rings(an, bn, rn);
      fetched = true;
      if (staged) {
        const double w = upstream ? upstream[i] : 1.0;
        // boxes apart: no crossings and no midpoint inside the other polygon
        const float x0 = fmaxf(ext[0].x, ext[1].x), x1 = fminf(ext[0].z, ext[1].z);
        const float y0 = fmaxf(ext[0].y, ext[1].y), y1 = fminf(ext[0].w, ext[1].w);
        if (!(x0 > x1 || y0 > y1)) {
          Poly A{base.ring_vert, base.ring_hole, base.xy, rr[0], rr[1]};
          Poly B{over.ring_vert, over.ring_hole, over.xy, rr[2], rr[3]};
          const SlabGrid gy = slab_grid(y0, y1), gx = slab_grid(x0, x1);
          if (V == kBwdOneV || (kMixed && nv[0] + nv[1] <= kBwdOneV))
            pair_boundary<false, true>(W, ext, nv[0], nv[1], gy, gx, w, grad_base, grad_over, vb[0], vb[1], A, B, 0.0,
                                       0.0, nullptr);
          else
            pair_boundary<false, false>(W, ext, nv[0], nv[1], gy, gx, w, grad_base, grad_over, vb[0], vb[1], A, B,
                                        0.0, 0.0, nullptr);
        }
      } else if (PL.defer && (V != kBwdMidV || max(nv[0], nv[1]) <= kBwdLargeV)) {
        if ((threadIdx.x & 31) == 0) PL.defer[atomicAdd(PL.defer_count, 1ull)] = (int32_t)i;
      } else if (V > kBwdOneV) {  // all that is listed for the smallest stage fits
        const double w = upstream ? upstream[i] : 1.0;
        Poly A{base.ring_vert, base.ring_hole, base.xy, rr[0], rr[1]};
        Poly B{over.ring_vert, over.ring_hole, over.xy, rr[2], rr[3]};
        bwd_pair_global(A, B, w, grad_base, grad_over);
      }
    }
    if (!fetched) rings(an, bn, rn);
    i = in;
    a = an;
    b = bn;
    for (int q = 0; q < 4; q++) rr[q] = rn[q];
    __syncwarp();
  }
  if constexpr (V == kBwdOneV) cudaGridDependencySynchronize();  // the next stage waits for this one alone
}

// Forward: one warp per pair, staged as in the backward.  A pair gets its
// area from pair_boundary's area mode when every crossing is clean and the
// crossing error bound stays below kFwdTol of the area; every other pair
// (polygons above V vertices or 31 rings, unclean crossings, slivers
// whose area the bound does not pin to kFwdTol, ids out of range) is listed in
// fb[] for the GPC clip.  GPC intersects the same edges, so for a clean pair
// the two areas differ only by where each side rounds the crossing vertices:
// a vertex moves by at most ~2 eps max|coordinate| / sin(angle), which moves
// the area by that times the crossing edges' lengths.  pair_boundary sums
// (|r|_1 + |s|_1) / sin over the crossings as seen from both edges (each
// crossing twice, and 1-norms, which are at least the lengths), so
// 2 eps max|coordinate| times the sum bounds the difference; a pair is kept
// when that is below kFwdTol of its area, ten times inside the 1e-9 the
// forward promises.
constexpr double kFwdTol = 1e-10;

// Pairs the last forward call listed for the GPC clip (prt_area_fwd_fallbacks).
std::atomic<int64_t> g_fwd_fallbacks{0};

// ---- pairs of tiny polygons: one thread each -----------------------------------
// Two polygons of one ring and 3 to kTinyV vertices (parcels, map tiles) have too
// few edges for a warp (4-6-vertex parcels filled 10 of its 32 lanes, and staging
// them cost more than their crossings).  One thread takes such a pair and
// intersects every pair of edges once, for both: with the edge p + t r of A
// and a + u s of B, t and u are the crossing seen from A's and from B's side, bit
// for bit what the two passes of pair_boundary compute.  B's vertices and
// per-edge sums stay in registers, A's vertices (and in gradient mode its
// gradient, until the pair is known to be clean) in shared memory.  The other
// pairs are listed for the staged kernels, the unclean ones too in gradient
// mode; in area mode those go to the GPC clip like theirs.  Of the pairs that are
// left, those of up to kBwdOneV vertices together have a stage of their own in
// gradient mode (100k pairs of 9-16 vertices: 364 us -> 295 us; 20k of equal
// 4-6-vertex parcels, all unclean, 180 -> 120).
constexpr int kTinyV = 8;
constexpr int kTinyBlock = 128;
// A thread takes 15-25 us for its pair however few there are.  Up to kFewPairs
// pairs, two or three waves of warps, every pair starts in the 64-vertex stage (1,000
// pairs of 4-6 vertices: backward 44 -> 31 us; from some 10,000 on the threads are as
// fast), and up to kOnePairWave, one wave of the 256-vertex stage, what does not
// fit goes straight to that.
constexpr int64_t kFewPairs = 8192, kOnePairWave = (int64_t)kSMs * 8;

// Appends i to a list for the threads of the block that ask (one atomic per
// block: when no pair is tiny, every one of them is listed).
__device__ __forceinline__ void append_pair(bool ask, int64_t i, int32_t *list, unsigned long long *count,
                                            unsigned *s_count, unsigned long long *s_base) {
  const unsigned who = __ballot_sync(kFullMask, ask);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_count[warp] = __popc(who);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned total = 0;
    for (int w = 0; w < kTinyBlock / 32; w++) total += s_count[w];
    *s_base = total ? atomicAdd(count, (unsigned long long)total) : 0ull;
  }
  __syncthreads();
  unsigned long long at = *s_base;
  for (int w = 0; w < warp; w++) at += s_count[w];
  if (ask) list[at + __popc(who & ((1u << lane) - 1u))] = (int32_t)i;
  __syncthreads();
}

// A polygon's rings, first vertex and vertices; whether a thread can take it, and
// then its ring's hole flag.
__device__ __forceinline__ bool tiny_ring(const LayerDev &L, int64_t poly, int64_t *rings, int64_t *v0, int64_t *nv,
                                          bool *hole) {
  const int64_t r = L.poly_ring[poly], e = L.poly_ring[poly + 1];
  *rings = e - r;
  *v0 = L.ring_vert[r];
  *nv = L.ring_vert[e] - *v0;
  if (e != r + 1 || *nv < 3 || *nv > kTinyV) return false;
  *hole = L.ring_hole && L.ring_hole[r];
  return true;
}

template <bool kArea>
struct TinySmem {
  double x[kTinyV][kTinyBlock], y[kTinyV][kTinyBlock];  // A's vertices, a column per thread
  double gx[kArea ? 1 : kTinyV][kTinyBlock], gy[kArea ? 1 : kTinyV][kTinyBlock];
};

// 200k parcels (471k pairs), the kernel alone: forward 85 us, backward 105 against 535
// and 604 with a warp each.  The whole call: 120 us backward with 3 blocks per SM, 132
// with 4 and 186 with 5; 103 us forward with 4, 107 and 123 with 3 and 5.
template <bool kArea>
__global__ void __launch_bounds__(kTinyBlock, kArea ? 4 : 3) area_tiny_kernel(
    const int32_t *__restrict__ pa, const int32_t *__restrict__ pb, int64_t n, LayerDev base, LayerDev over,
    const double *__restrict__ upstream, double *grad_base, double *grad_over, double *__restrict__ area,
    int32_t *__restrict__ fb, unsigned long long *__restrict__ fb_count, int32_t *__restrict__ defer,
    unsigned long long *__restrict__ defer_count, int32_t *__restrict__ one, unsigned long long *__restrict__ one_count) {
  __shared__ TinySmem<kArea> S;
  __shared__ unsigned s_count[kTinyBlock / 32];
  __shared__ unsigned long long s_base;
  const int tid = threadIdx.x;
  const int64_t i = blockIdx.x * (int64_t)kTinyBlock + tid;
  int64_t va = 0, vb = 0;
  int na = 0, nb = 0;
  bool ha = false, hb = false;
  bool mine = false, few = false;  // this thread takes the pair; the smallest stage can
  if (i < n) {
    const int64_t a = pa[i], b = pb[i];
    if (a >= 0 && a < base.n_poly && b >= 0 && b < over.n_poly) {
      int64_t ra, rb, ma, mb;
      const bool ta = tiny_ring(base, a, &ra, &va, &ma, &ha), tb = tiny_ring(over, b, &rb, &vb, &mb, &hb);
      mine = ta && tb;
      few = ra <= 31 && rb <= 31 && ma + mb <= kBwdOneV;
      na = (int)ma;
      nb = (int)mb;
    }
  }
  bool clean = true;
  double bound = 0.0, area2 = 0.0;
  if (mine) {
    double bx[kTinyV], by[kTinyV];
    double cmax = 0.0, sa = 0.0, sb = 0.0;
    double lox = 0.0, loy = 0.0, hix = 0.0, hiy = 0.0;  // A's box
    for (int k = 0; k < na; k++) {
      const double x = base.xy[2 * (va + k)], y = base.xy[2 * (va + k) + 1];
      S.x[k][tid] = x;
      S.y[k][tid] = y;
      lox = k ? fmin(lox, x) : x;
      loy = k ? fmin(loy, y) : y;
      hix = k ? fmax(hix, x) : x;
      hiy = k ? fmax(hiy, y) : y;
    }
    cmax = fmax(fmax(fabs(lox), fabs(loy)), fmax(fabs(hix), fabs(hiy)));
    double blx = 0.0, bly = 0.0, bhx = 0.0, bhy = 0.0;
#pragma unroll
    for (int k = 0; k < kTinyV; k++) {
      bx[k] = by[k] = 0.0;
      if (k < nb) {
        bx[k] = over.xy[2 * (vb + k)];
        by[k] = over.xy[2 * (vb + k) + 1];
        blx = k ? fmin(blx, bx[k]) : bx[k];
        bly = k ? fmin(bly, by[k]) : by[k];
        bhx = k ? fmax(bhx, bx[k]) : bx[k];
        bhy = k ? fmax(bhy, by[k]) : by[k];
      }
    }
    cmax = fmax(cmax, fmax(fmax(fabs(blx), fabs(bly)), fmax(fabs(bhx), fabs(bhy))));
    // boxes apart: no crossing, no point of one inside the other (the boxes leave
    // NaN coordinates out, as the staged kernels' do; of a pair that is not apart
    // they are not clean below)
    const bool apart = lox > bhx || hix < blx || loy > bhy || hiy < bly;
    if (!apart) {
      for (int k = 0; k < na; k++) {
        const int l = k + 1 == na ? 0 : k + 1;
        sa += S.x[k][tid] * S.y[l][tid] - S.x[l][tid] * S.y[k][tid];
      }
#pragma unroll
      for (int k = 0; k < kTinyV; k++)
        if (k < nb) {
          const bool last = k + 1 == nb;
          const double ex = last ? bx[0] : bx[k + 1 < kTinyV ? k + 1 : 0], ey = last ? by[0] : by[k + 1 < kTinyV ? k + 1 : 0];
          sb += bx[k] * ey - ex * by[k];
        }
      // material on the left: CCW outer rings and CW holes
      const bool la = (sa >= 0.0) != ha, lb = (sb >= 0.0) != hb;
      const double sgna = la ? 1.0 : -1.0, sgnb = lb ? 1.0 : -1.0;
      const double w = !kArea && upstream ? upstream[i] : 1.0;
      const double ox = S.x[0][tid], oy = S.y[0][tid];  // the pair-local origin
      // per edge of B: sums of sign u and sign u^2, and crossings (low half) and
      // signs (high half) as 4-bit fields, biased by 8
      double c1b[kTinyV], c2b[kTinyV];
#pragma unroll
      for (int k = 0; k < kTinyV; k++) c1b[k] = c2b[k] = 0.0;
      uint32_t mb = 0, c0b = 0x88888888u;
      double ufirst = 1.0;  // first crossing of B's edge 0
      double err = 0.0;
      bool st = false;  // inside state at the start of A's edge k
      double cx = 0.0, cy = 0.0;  // what the edge before gives to A's vertex k
      for (int k = 0; k < na && clean; k++) {
        const int l = k + 1 == na ? 0 : k + 1;
        const double px = S.x[k][tid], py = S.y[k][tid], qx = S.x[l][tid], qy = S.y[l][tid];
        const double rx = qx - px, ry = qy - py;
        const double rl = fabs(rx) + fabs(ry);
        double c1 = 0.0, c2 = 0.0, tfirst = 1.0;
        int m = 0, c0 = 0;
#pragma unroll
        for (int e = 0; e < kTinyV; e++) {
          if (e >= nb) break;
          const bool last = e + 1 == nb;
          const double ax = bx[e], ay = by[e];
          const double sx = (last ? bx[0] : bx[e + 1 < kTinyV ? e + 1 : 0]) - ax;
          const double sy = (last ? by[0] : by[e + 1 < kTinyV ? e + 1 : 0]) - ay;
          const double den = rx * sy - ry * sx;
          const double apx = ax - px, apy = ay - py;
          const double tn = apx * sy - apy * sx;
          const double un = apx * ry - apy * rx;
          if (den == 0.0) {
            // collinear edges whose boxes meet
            if ((tn == 0.0 || un == 0.0) && fmin(ax, ax + sx) <= fmax(px, qx) && fmin(px, qx) <= fmax(ax, ax + sx) &&
                fmin(ay, ay + sy) <= fmax(py, qy) && fmin(py, qy) <= fmax(ay, ay + sy))
              clean = false;
            continue;
          }
          // t = tn / den and u = un / den, with the signs of den folded in
          const double d = fabs(den), tol = 1e-9 * d;
          const double tt = den > 0.0 ? tn : -tn, uu = den > 0.0 ? un : -un;
          if (tt < -tol || tt > d + tol || uu < -tol || uu > d + tol) continue;
          const double sl = fabs(sx) + fabs(sy);
          if (!(tt > tol && tt < d - tol && uu > tol && uu < d - tol && d > 1e-6 * rl * sl)) {
            clean = false;
            continue;
          }
          if constexpr (kArea) err += 2.0 * ((rl + sl) * rl * sl / d);  // seen from both edges
          const double t = tn / den, u = un / den;
          const bool out_b = (den > 0.0) == lb;  // A's edge leaves B here
          const bool out_a = (den < 0.0) == la;  // B's edge leaves A
          const double ts = out_b ? -t : t, us = out_a ? -u : u;
          c0 += out_b ? -1 : 1;
          c1 += ts;
          if constexpr (!kArea) c2 += ts * t;
          tfirst = fmin(tfirst, t);
          m++;
          c0b += out_a ? 0u - (1u << (4 * e)) : 1u << (4 * e);
          mb ^= 1u << e;
          c1b[e] += us;
          if constexpr (!kArea) c2b[e] += us * u;
          if (e == 0) ufirst = fmin(ufirst, u);
        }
        if (k == 0) {
          // the ring's first piece by its midpoint
          const double mx = px + 0.5 * tfirst * rx, my = py + 0.5 * tfirst * ry;
          bool in = false;
#pragma unroll
          for (int e = 0; e < kTinyV; e++) {
            if (e >= nb) break;
            const bool last = e + 1 == nb;
            const double ax = bx[e], ay = by[e];
            const double ex = last ? bx[0] : bx[e + 1 < kTinyV ? e + 1 : 0], ey = last ? by[0] : by[e + 1 < kTinyV ? e + 1 : 0];
            if ((ay > my) != (ey > my) && mx < ax + (my - ay) * (ex - ax) / (ey - ay)) in = !in;
          }
          st = in;
        }
        const bool end = st != ((m & 1) != 0);
        if ((int)st + c0 != (int)end) clean = false;
        st = end;
        const double s1 = end ? 1.0 : 0.0;
        if constexpr (kArea) {
          area2 += sgna * (s1 - c1) * ((px - ox) * ry - (py - oy) * rx);
        } else {
          const double it = 0.5 * (s1 - c2), i1 = (s1 - c1) - it;
          const double nx = w * sgna * ry, ny = -w * sgna * rx;
          S.gx[k][tid] = cx + nx * i1;
          S.gy[k][tid] = cy + ny * i1;
          cx = nx * it;
          cy = ny * it;
        }
      }
      if constexpr (!kArea) {
        S.gx[0][tid] += cx;
        S.gy[0][tid] += cy;
      }
      // B's edges, from their sums
      {
        const double dx = bx[1] - bx[0], dy = by[1] - by[0];
        const double mx = bx[0] + 0.5 * ufirst * dx, my = by[0] + 0.5 * ufirst * dy;
        bool in = false;
        for (int k = 0; k < na; k++) {
          const int l = k + 1 == na ? 0 : k + 1;
          const double ax = S.x[k][tid], ay = S.y[k][tid], ex = S.x[l][tid], ey = S.y[l][tid];
          if ((ay > my) != (ey > my) && mx < ax + (my - ay) * (ex - ax) / (ey - ay)) in = !in;
        }
        st = in;
      }
      uint32_t ends = 0;  // inside state at the edges' ends
#pragma unroll
      for (int e = 0; e < kTinyV; e++) {
        if (e >= nb) break;
        const bool end = st != ((mb >> e & 1u) != 0);
        if ((int)st + (int)(c0b >> (4 * e) & 15u) - 8 != (int)end) clean = false;
        st = end;
        ends |= (end ? 1u : 0u) << e;
      }
      if constexpr (kArea) {
#pragma unroll
        for (int e = 0; e < kTinyV; e++) {
          if (e >= nb) break;
          const bool last = e + 1 == nb;
          const double rx = (last ? bx[0] : bx[e + 1 < kTinyV ? e + 1 : 0]) - bx[e];
          const double ry = (last ? by[0] : by[e + 1 < kTinyV ? e + 1 : 0]) - by[e];
          const double s1 = ends >> e & 1u ? 1.0 : 0.0;
          area2 += sgnb * (s1 - c1b[e]) * ((bx[e] - ox) * ry - (by[e] - oy) * rx);
        }
        bound = 2.0 * 2.220446049250313e-16 * cmax * err;
      } else if (clean) {
        for (int k = 0; k < na; k++) {
          const double x = S.gx[k][tid], y = S.gy[k][tid];
          if (x != 0.0 || y != 0.0) {
            atomicAdd(&grad_base[2 * (va + k)], x);
            atomicAdd(&grad_base[2 * (va + k) + 1], y);
          }
        }
        double fx = 0.0, fy = 0.0;  // vertex 0's own part
        cx = cy = 0.0;
#pragma unroll
        for (int e = 0; e < kTinyV; e++) {
          if (e >= nb) break;
          const bool last = e + 1 == nb;
          const double rx = (last ? bx[0] : bx[e + 1 < kTinyV ? e + 1 : 0]) - bx[e];
          const double ry = (last ? by[0] : by[e + 1 < kTinyV ? e + 1 : 0]) - by[e];
          const double s1 = ends >> e & 1u ? 1.0 : 0.0;
          const double it = 0.5 * (s1 - c2b[e]), i1 = (s1 - c1b[e]) - it;
          const double nx = w * sgnb * ry, ny = -w * sgnb * rx;
          const double x = cx + nx * i1, y = cy + ny * i1;
          if (e == 0) {
            fx = x;
            fy = y;
          } else if (x != 0.0 || y != 0.0) {
            atomicAdd(&grad_over[2 * (vb + e)], x);
            atomicAdd(&grad_over[2 * (vb + e) + 1], y);
          }
          cx = nx * it;
          cy = ny * it;
        }
        fx += cx;
        fy += cy;
        if (fx != 0.0 || fy != 0.0) {
          atomicAdd(&grad_over[2 * vb], fx);
          atomicAdd(&grad_over[2 * vb + 1], fy);
        }
      }
    }
  }
  if constexpr (kArea) {
    const double ar = 0.5 * area2;
    const bool keep = mine && clean && bound <= kFwdTol * fabs(ar);
    if (keep) area[i] = ar;
    append_pair(mine && !keep, i, fb, fb_count, s_count, &s_base);
    append_pair(i < n && !mine, i, defer, defer_count, s_count, &s_base);
  } else {
    const bool left = i < n && !(mine && clean);
    append_pair(left && few, i, one, one_count, s_count, &s_base);
    append_pair(left && !few, i, defer, defer_count, s_count, &s_base);
  }
}

// V = 64: 5 blocks of 4 warps per SM (96 registers: a few spills, 10% faster
// than 4 blocks at 1M pairs of 16-64-vertex stars).
template <int V>
__global__ void __launch_bounds__(32 * bwd_warps(V), V <= kBwdSmallV || V > kBwdMidV ? 5 : 4) area_fwd_kernel(
    const int32_t *__restrict__ pa, const int32_t *__restrict__ pb, int64_t n, LayerDev base, LayerDev over,
    double *__restrict__ area, int32_t *__restrict__ fb, unsigned long long *__restrict__ fb_count, PairList PL) {
  __shared__ BwdPair<V> sm[bwd_warps(V)];
  BwdPair<V> &W = sm[threadIdx.x >> 5];
  BwdPoly<V> *M = W.poly;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  cudaGridDependencySynchronize();
  const int64_t items = list_items(PL, n);
  auto fallback = [&](int64_t i) {
    if (lane == 0) fb[atomicAdd(fb_count, 1ull)] = (int32_t)i;
  };
  for (int64_t k = warp; k < items; k += nw) {
    const int64_t i = PL.sel ? PL.sel[k] : k;
    if (i < 0 || i >= n) continue;
    const int64_t a = pa[i], b = pb[i];
    if (a < 0 || a >= base.n_poly || b < 0 || b >= over.n_poly) {
      fallback(i);  // the clip reports the bad id
      continue;
    }
    const int64_t ra0 = base.poly_ring[a], ra1 = base.poly_ring[a + 1];
    const int64_t rb0 = over.poly_ring[b], rb1 = over.poly_ring[b + 1];
    int nv[2];
    int64_t vb[2];
    float4 ext[2];
    const bool staged = bwd_load_pair(base, ra0, ra1, over, rb0, rb1, M, nv, vb, ext);
    if (!staged) {
      if (PL.defer) {
        if (lane == 0) PL.defer[atomicAdd(PL.defer_count, 1ull)] = (int32_t)i;
      } else {
        fallback(i);
      }
      __syncwarp();
      continue;
    }
    const float x0 = fmaxf(ext[0].x, ext[1].x), x1 = fminf(ext[0].z, ext[1].z);
    const float y0 = fmaxf(ext[0].y, ext[1].y), y1 = fminf(ext[0].w, ext[1].w);
    if (x0 > x1 || y0 > y1 || nv[0] == 0 || nv[1] == 0) {
      // boxes apart: no crossing, no point of one inside the other
      if (lane == 0) area[i] = 0.0;
      __syncwarp();
      continue;
    }
    const SlabGrid gy = slab_grid(y0, y1), gx = slab_grid(x0, x1);
    Poly A{base.ring_vert, base.ring_hole, base.xy, ra0, ra1};
    Poly B{over.ring_vert, over.ring_hole, over.xy, rb0, rb1};
    AreaSum acc{0.0, 0.0};
    const double ox = M[0].x[0], oy = M[0].y[0];  // the pair-local origin
    const bool ok = pair_boundary<true, false>(W, ext, nv[0], nv[1], gy, gx, 1.0, nullptr, nullptr, vb[0], vb[1], A, B,
                                               ox, oy, &acc);
    if (ok) {
      double a2 = acc.area, er = acc.err;
      for (int o = 16; o; o >>= 1) {
        a2 += __shfl_xor_sync(kFullMask, a2, o);
        er += __shfl_xor_sync(kFullMask, er, o);
      }
      const float cmax = fmaxf(fmaxf(fmaxf(fabsf(ext[0].x), fabsf(ext[0].y)), fmaxf(fabsf(ext[0].z), fabsf(ext[0].w))),
                               fmaxf(fmaxf(fabsf(ext[1].x), fabsf(ext[1].y)), fmaxf(fabsf(ext[1].z), fabsf(ext[1].w))));
      const double bound = 2.0 * 2.220446049250313e-16 * (double)cmax * er;
      const double ar = 0.5 * a2;
      if (bound <= kFwdTol * fabs(ar)) {
        if (lane == 0) area[i] = ar;
      } else {
        fallback(i);
      }
    } else {
      fallback(i);
    }
    __syncwarp();
  }
}

__global__ void gather_pairs_kernel(const int32_t *__restrict__ fb, int64_t m, const int32_t *__restrict__ pa,
                                    const int32_t *__restrict__ pb, int32_t *__restrict__ qa,
                                    int32_t *__restrict__ qb) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
    qa[k] = pa[fb[k]];
    qb[k] = pb[fb[k]];
  }
}

__global__ void scatter_area_kernel(const int32_t *__restrict__ fb, int64_t m, const double *__restrict__ src,
                                    double *__restrict__ area) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
    area[fb[k]] = src[k];
}

// Exactly the resident blocks (each warp loops over pairs): no tail wave.
int area_blocks(int64_t n_pairs, int threads, const void *kernel, std::atomic<int> &per_sm) {
  int b = per_sm.load(std::memory_order_relaxed);
  if (b == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, 0) != cudaSuccess || b < 1) {
      cudaGetLastError();
      b = 4;
    }
    per_sm.store(b, std::memory_order_relaxed);
  }
  return grid_for(n_pairs * 32, threads, b);
}

template <int V>
cudaError_t launch_area_fwd(const int32_t *pa, const int32_t *pb, int64_t n, const LayerDev &base, const LayerDev &over,
                            double *area, int32_t *fb, unsigned long long *fb_count, const PairList &PL, cudaStream_t s) {
  const int threads = 32 * bwd_warps(V);
  static std::atomic<int> per_sm{0};
  return launch_dependent(area_fwd_kernel<V>, area_blocks(n, threads, (const void *)area_fwd_kernel<V>, per_sm), threads,
                          0, s, pa, pb, n, base, over, area, fb, fb_count, PL);
}

template <int V, bool kMixed = false>
cudaError_t launch_area_bwd(const int32_t *pa, const int32_t *pb, int64_t n, const LayerDev &base, const LayerDev &over,
                            const double *up, double *gb, double *go, const PairList &PL, cudaStream_t s) {
  const int threads = 32 * bwd_warps(V);
  static std::atomic<int> per_sm{0};
  return launch_dependent(area_bwd_kernel<V, kMixed>,
                          area_blocks(n, threads, (const void *)area_bwd_kernel<V, kMixed>, per_sm), threads, 0, s, pa,
                          pb, n, base, over, up, gb, go, PL);
}

}  // namespace
}  // namespace prt

using namespace prt;

extern "C" {

int prt_area_fwd(const int32_t *d_pair_a, const int32_t *d_pair_b, int64_t n_pairs, const prt_layer *base,
                 const prt_layer *overlay, double *d_area, void *stream) {
  PRT_CHECK(base && overlay && (n_pairs == 0 || (d_area && d_pair_a && d_pair_b)), PRT_ERR_INVALID,
            "NULL argument");
  PRT_CHECK(n_pairs >= 0 && n_pairs < (1ll << 31), PRT_ERR_INVALID, "n_pairs=%lld", (long long)n_pairs);
  if (n_pairs == 0) return PRT_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // boundary integral for the clean pairs, the list of the others; pairs
  // with a polygon too large for one stage's staging go to the next
  unsigned char *scr = nullptr;
  int rc = dmalloc(reinterpret_cast<void **>(&scr), 64 + 16 * (size_t)n_pairs, s);
  if (rc) return rc;
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(scr);  // fallbacks, then the three stage lists
  int32_t *fb = reinterpret_cast<int32_t *>(scr + 64);
  int32_t *small = fb + n_pairs, *mid = small + n_pairs, *large = mid + n_pairs;
  cudaError_t e = cudaMemsetAsync(cnt, 0, 32, s);
  if (e == cudaSuccess) {
    PRT_PROF("area_fwd", s);
    const LayerDev A = layer_dev(base), B = layer_dev(overlay);
    if (n_pairs > kFewPairs) {
      area_tiny_kernel<true><<<(unsigned)((n_pairs + kTinyBlock - 1) / kTinyBlock), kTinyBlock, 0, s>>>(
          d_pair_a, d_pair_b, n_pairs, A, B, nullptr, nullptr, nullptr, d_area, fb, cnt, small, cnt + 1, nullptr,
          nullptr);
      e = cudaGetLastError();
    }
    PairList first = {nullptr, nullptr, mid, cnt + 2}, last = {mid, cnt + 2, nullptr, nullptr};
    if (n_pairs > kFewPairs) first = {small, cnt + 1, mid, cnt + 2};
    if (n_pairs > kOnePairWave) last = {large, cnt + 3, nullptr, nullptr};
    if (e == cudaSuccess) e = launch_area_fwd<kBwdSmallV>(d_pair_a, d_pair_b, n_pairs, A, B, d_area, fb, cnt, first, s);
    if (e == cudaSuccess && n_pairs > kOnePairWave)
      e = launch_area_fwd<kBwdMidV>(d_pair_a, d_pair_b, n_pairs, A, B, d_area, fb, cnt,
                                    PairList{mid, cnt + 2, large, cnt + 3}, s);
    if (e == cudaSuccess) e = launch_area_fwd<kBwdLargeV>(d_pair_a, d_pair_b, n_pairs, A, B, d_area, fb, cnt, last, s);
  }
  unsigned long long m = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&m, cnt, 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    dfree(scr, s);
    return cuda_status(e, "area forward");
  }
  g_fwd_fallbacks.store((int64_t)m);
  if (m > 0) {
    // the listed pairs: GPC clip, area of its result (area-only mode)
    int32_t *q = nullptr;
    double *ar = nullptr;
    rc = dalloc(&q, 2 * m, s);
    if (!rc) rc = dalloc(&ar, m, s);
    if (!rc) {
      {
        PRT_PROF("gather_pairs", s);
        gather_pairs_kernel<<<grid_for((int64_t)m, 256, 8), 256, 0, s>>>(fb, (int64_t)m, d_pair_a, d_pair_b, q,
                                                                           q + m);
      }
      PairSrc S;
      memset(&S, 0, sizeof S);
      S.pa = q;
      S.pb = q + m;
      S.base = layer_dev(base);
      S.over = layer_dev(overlay);
      S.op = PRT_GPC_INT;
      rc = overlay_impl(S, (int64_t)m, PRT_SCHED_BATCHED, ar, s, nullptr);
    }
    if (!rc) {
      PRT_PROF("scatter_area", s);
      scatter_area_kernel<<<grid_for((int64_t)m, 256, 8), 256, 0, s>>>(fb, (int64_t)m, ar, d_area);
      e = cudaGetLastError();
      if (e != cudaSuccess) rc = cuda_status(e, "area scatter");
    }
    dfree(q, s);
    dfree(ar, s);
  }
  dfree(scr, s);
  return rc;
}

int prt_area_fwd_fallbacks(int64_t *h_count) {
  PRT_CHECK(h_count, PRT_ERR_INVALID, "NULL argument");
  *h_count = g_fwd_fallbacks.load();
  return PRT_OK;
}

int prt_area_bwd(const int32_t *d_pair_a, const int32_t *d_pair_b, int64_t n_pairs, const prt_layer *base,
                 const prt_layer *overlay, const double *d_upstream, double *d_grad_base, double *d_grad_overlay,
                 void *stream) {
  PRT_CHECK(base && overlay && (n_pairs == 0 || (d_grad_base && d_grad_overlay && d_pair_a && d_pair_b)),
            PRT_ERR_INVALID, "NULL argument");
  if (n_pairs == 0) return PRT_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // pairs that tiny polygons' threads leave, of few vertices together or more;
  // pairs with a polygon too large for one stage's staging: listed by it, taken by
  // the next
  unsigned char *scr = nullptr;
  int rc = dmalloc(reinterpret_cast<void **>(&scr), 64 + 16 * (size_t)n_pairs, s);
  if (rc) return rc;
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(scr);  // the stages' lists
  int32_t *one = reinterpret_cast<int32_t *>(scr + 64);
  int32_t *small = one + n_pairs, *mid = small + n_pairs, *large = mid + n_pairs;
  cudaError_t e = cudaMemsetAsync(cnt, 0, 32, s);
  if (e == cudaSuccess) {
    PRT_PROF("area_bwd", s);
    const LayerDev A = layer_dev(base), B = layer_dev(overlay);
    PairList last = {mid, cnt + 1, nullptr, nullptr};
    if (n_pairs > kOnePairWave) last = {large, cnt + 2, nullptr, nullptr};
    if (n_pairs > kFewPairs) {
      area_tiny_kernel<false><<<(unsigned)((n_pairs + kTinyBlock - 1) / kTinyBlock), kTinyBlock, 0, s>>>(
          d_pair_a, d_pair_b, n_pairs, A, B, d_upstream, d_grad_base, d_grad_overlay, nullptr, nullptr, nullptr, small,
          cnt, one, cnt + 3);
      e = cudaGetLastError();
      if (e == cudaSuccess)
        e = launch_area_bwd<kBwdSmallV>(d_pair_a, d_pair_b, n_pairs, A, B, d_upstream, d_grad_base, d_grad_overlay,
                                        PairList{small, cnt, mid, cnt + 1}, s);
      if (e == cudaSuccess)
        e = launch_area_bwd<kBwdOneV>(d_pair_a, d_pair_b, n_pairs, A, B, d_upstream, d_grad_base, d_grad_overlay,
                                      PairList{one, cnt + 3, nullptr, nullptr}, s);
    } else {
      e = launch_area_bwd<kBwdSmallV, true>(d_pair_a, d_pair_b, n_pairs, A, B, d_upstream, d_grad_base, d_grad_overlay,
                                            PairList{nullptr, nullptr, mid, cnt + 1}, s);
    }
    if (e == cudaSuccess && n_pairs > kOnePairWave)
      e = launch_area_bwd<kBwdMidV>(d_pair_a, d_pair_b, n_pairs, A, B, d_upstream, d_grad_base, d_grad_overlay,
                                    PairList{mid, cnt + 1, large, cnt + 2}, s);
    if (e == cudaSuccess)
      e = launch_area_bwd<kBwdLargeV>(d_pair_a, d_pair_b, n_pairs, A, B, d_upstream, d_grad_base, d_grad_overlay, last,
                                      s);
  }
  dfree(scr, s);
  if (e != cudaSuccess) return cuda_status(e, "area backward");
  return PRT_OK;
}

}  // extern "C"
