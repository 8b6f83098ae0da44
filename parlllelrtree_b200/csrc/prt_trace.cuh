// Overlay of a pair in general position by tracing, with the result that the
// scanbeam clippers (prt_gpc.cuh, prt_wgpc.cuh) give, bit for bit.
//
// GPC sweeps the pair beam by beam (a beam: two neighbouring vertex ys), a chain
// of dependent steps per beam however little happens in it.  When nothing
// degenerate happens anywhere, its result follows from the crossings alone:
//  * the vertices of A ∩ B are the input vertices inside the other polygon, as
//    they are, and the crossings, and a crossing's coordinates are a function of
//    its two edges and the beam that it lies in (the edges' x at the beam's two
//    ys, build_intersection_table, GPC:1309-1471);
//  * the boundary runs along A where A is inside B and along B where B is inside
//    A (outside for a union, and of a difference along B backwards) and changes
//    over at every crossing, so the contours are cycles of runs of consecutive
//    vertices between crossings; an exclusive or keeps every run, and at a crossing
//    one contour ends below and another starts above;
//  * GPC's vertex lists grow to the left and right and are joined at maxima, so a
//    contour comes out cut at its highest vertex: that vertex is the last one
//    written of an outer contour and the first one of a hole;
//  * contours are listed newest first, by the local minimum that opened the
//    output polygon which survived the joins: at an outer maximum the polygon of
//    the edge on the right survives, at a hole's maximum too, which is the
//    boundary's incoming side at the first and its outgoing side at the second.
//  Equal ys count left to right, as the clipper works through a scanline.
// General position is checked, not assumed: any two edges that share a y range are
// further apart at both ends of it than rounding can move them (or cross properly,
// with the same distance at the crossing's beam), edges that meet in a local
// extremum included, at the vertex y next to it.  The distance between two edges is
// linear in y, so that covers every beam.  No vertex lies on a horizontal edge, no
// two horizontal edges follow each other (GPC drops the vertex between them), and no y
// is -0.  A polygon that crosses or touches itself fails the check too.  A pair that
// fails it, or that has more vertices, rings or crossings than there is room for, is
// left to the scanbeam clippers.
//
// A block per pair, everything between the input and the result in shared memory,
// vertices in 16-bit indices so that two pairs of 4,160 vertices share an SM.  What
// bounds it is the search for edges that meet: its lists are short (13 edges on
// average for rings of 4,096 vertices) but scattered in shared memory.  Measured
// against the scanbeam clippers alone: 21,000 star pairs of 16 to 64 vertices 2,435
// -> 290 us, 40,000 pairs of 8 to 8,192 vertices 162 -> 10.2 ms (all traced; a pair
// of 4,300 vertices that is left costs 16 ms, as the beams of one pair are a chain).
#pragma once
#include "prt_gpc.cuh"

namespace prt {
namespace trace {

constexpr int kMaxRings = 32;
constexpr int kLast = 0x8000;
// Smallest |y| of a vertex that is not 0, 2^-432 or 1e-130: two ys are then 1e-146
// apart or equal, so that neither the slopes nor the buckets per unit of y below
// overflow, and what a product of an x and a y difference loses to underflow is far
// below the margin.  -0 is no y either: of two zeros on a scanline the clipper writes
// one for all, and the y difference of a horizontal edge between them may be -0, its
// slope then -inf.  (In integers: two comparisons of doubles per vertex, and one of
// signs per tie, cost the 60,000 stars' 2.19 ms 4%.)
constexpr int kLeastY = (1023 - 432) << 20;  // a double's high word
__device__ __forceinline__ bool y_allowed(double y) {
  const int hi = __double2hiint(y);
  return (hi & 0x7fffffff) >= kLeastY || (hi | __double2loint(y)) == 0;
}
// Coordinates stay below this: products of two differences do not overflow.
constexpr double kMostXY = 1e150;

template <int NT>
__device__ __forceinline__ void bsync() {
  if constexpr (NT == 32) __syncwarp();
  else __syncthreads();
}

// Whether v holds on any thread of the block: the same answer on all of them, so
// that they leave together.
template <int NT>
__device__ __forceinline__ bool bany(bool v) {
  if constexpr (NT == 32) {
    const bool any = __any_sync(0xffffffffu, v);
    __syncwarp();
    return any;
  } else {
    return __syncthreads_or(v);
  }
}

// Room for one class of pairs: NT threads per pair; at most kVerts vertices and
// kCross crossings; 2^kSlabShift vertex ys per slab of the edge search; kList edges over
// all slabs, and nodes over all contours.
template <int NT_, int kVerts_, int kCross_, int kSlabShift_, int kList_, int kBlocks_, int kTwo_>
struct Class {
  static constexpr int NT = NT_, kVerts = kVerts_, kCross = kCross_, kSlabShift = kSlabShift_, kList = kList_;
  static constexpr int kBlocks = kBlocks_;  // resident per SM
  static constexpr int kTwo = kTwo_;        // 1: exclusive or (an instantiation of its own costs the others nothing)
  static constexpr int kSlabs = (kVerts >> kSlabShift) + 1;
  static constexpr int kContours = kCross / 2 + kMaxRings;
  static_assert(kList >= kVerts && kCross >= 2 * kMaxRings && kCross < 4095 && kVerts <= kLast, "limits");
};

template <typename C>
struct Smem {
  double sy[C::kVerts];  // vertex ys, sorted
  double vx[C::kVerts];
  double cx[C::kCross], cy[C::kCross], crel[C::kCross];  // crossings: coordinates, y above the beam's lower y
  float ctol[C::kCross];  // what crel may be off by
  double red[4][16];
  double rbb[kMaxRings][4];
  const double *rxy[kMaxRings];  // ring's vertices in global memory
  int64_t cbase, vbase;
  uint32_t rep[C::kContours];  // key of the minimum that a contour is listed by
  uint16_t head[C::kContours], len[C::kContours], place[C::kContours], off[C::kContours];
  uint16_t top[C::kContours];  // position of the highest node
  int slab0[C::kSlabs + 1];
  int rstart[kMaxRings + 1];
  uint16_t runoff[C::kCross], cnt[C::kCross];
  uint16_t rank[C::kVerts];      // of vertex v among the sorted ys
  uint16_t list[C::kList];       // vertices in y order; then edges per slab; then the contours' nodes
  uint16_t ce[2][C::kCross];     // crossing's edge of A and of B
  uint16_t beam[C::kCross], ord[C::kCross], seq[2][C::kCross], pos[2][C::kCross], next[C::kCross];
  uint8_t ring[C::kVerts];
  uint8_t aleft[C::kCross], out[C::kCross], cyc[C::kCross];
  uint8_t rside[kMaxRings], mat[kMaxRings], hit[kMaxRings];
  uint8_t hole[C::kContours];
  uint32_t queue[C::NT / 32][64];
  int ncross, ncont, nodes;
  unsigned long long ticket, best;
};

template <typename C>
struct Pair {
  Smem<C> &S;
  int n;
  double margin, least;
  bool convex;
  // an exclusive or has two nodes per crossing: 2c where contours end below it,
  // 2c + 1 where they start above
  static constexpr int two = C::kTwo;
  __device__ __forceinline__ int crossing(int node) const { return (node & 0x7fff) >> two; }
  __device__ __forceinline__ bool up(int v) const { return S.rank[nxt(v)] > S.rank[v]; }
  __device__ __forceinline__ double x(int v) const { return S.vx[v]; }
  __device__ __forceinline__ double y(int v) const { return S.sy[S.rank[v]]; }
  __device__ __forceinline__ int nxt(int v) const {
    const int r = S.ring[v];
    return v + 1 == S.rstart[r + 1] ? S.rstart[r] : v + 1;
  }
  __device__ __forceinline__ int prv(int v) const {
    const int r = S.ring[v];
    return v == S.rstart[r] ? S.rstart[r + 1] - 1 : v - 1;
  }
};

// An edge as GPC holds it: bottom, top, slope; ranks of its ends.
struct TEdge {
  double bx, by, tx, ty, dx;
  int v, w, rb, rt;  // start and end vertex, lower and upper rank
  bool up;
  __device__ __forceinline__ double at(double y) const { return y == ty ? tx : bx + dx * (y - by); }
};

template <typename C>
__device__ __forceinline__ TEdge edge_of(const Pair<C> &P, int v) {
  TEdge e;
  e.v = v;
  e.w = P.nxt(v);
  const int r1 = P.S.rank[e.v], r2 = P.S.rank[e.w];
  e.up = r2 > r1;
  e.rb = e.up ? r1 : r2;
  e.rt = e.up ? r2 : r1;
  const double x1 = P.x(e.v), x2 = P.x(e.w);
  e.bx = e.up ? x1 : x2;
  e.tx = e.up ? x2 : x1;
  e.by = P.S.sy[e.rb];
  e.ty = P.S.sy[e.rt];
  e.dx = (e.tx - e.bx) / (e.ty - e.by);  // horizontal: +inf, its left end is the lower one
  return e;
}

// The edge's ranks and its x range, widened by the margin.
template <typename C>
__device__ __forceinline__ void edge_box(const Pair<C> &P, int v, int &rb, int &rt, double &xlo, double &xhi) {
  const int w = P.nxt(v), r1 = P.S.rank[v], r2 = P.S.rank[w];
  rb = min(r1, r2);
  rt = max(r1, r2);
  const double x1 = P.x(v), x2 = P.x(w);
  xlo = (x1 < x2 ? x1 : x2) - P.margin;
  xhi = (x1 < x2 ? x2 : x1) + P.margin;
}

// Records the crossing of a and b; true when there is no room for it.
template <typename C>
__device__ __forceinline__ bool add_crossing(Smem<C> &S, const TEdge &a, const TEdge &b, double x, double y, double rel,
                                             double tol, int beam, bool a_left) {
  const int c = atomicAdd(&S.ncross, 1);
  if (c >= C::kCross) return true;
  const int ra = S.rside[S.ring[a.v]];
  S.cx[c] = x;
  S.cy[c] = y;
  S.crel[c] = rel;
  S.ctol[c] = __double2float_ru(tol);
  S.beam[c] = (uint16_t)beam;
  S.ce[ra][c] = (uint16_t)a.v;
  S.ce[1 - ra][c] = (uint16_t)b.v;
  S.aleft[c] = (ra == 0) == a_left;  // polygon 0's edge is on the left below
  return false;
}

// A horizontal edge and another one: no vertex may lie on it.
template <typename C>
__device__ bool test_horizontal(const Pair<C> &P, const TEdge &h, const TEdge &b) {
  Smem<C> &S = P.S;
  const double m = P.margin, y = h.by;
  if (b.by == b.ty) return true;  // their x ranges meet, as their ranks do
  if (h.w == b.v || b.w == h.v) return false;
  const double x = b.at(y);
  if (x < h.bx - m || x > h.tx + m) return false;
  if (b.by == y || b.ty == y || x - h.bx <= m || h.tx - x <= m) return true;
  if (S.rside[S.ring[h.v]] == S.rside[S.ring[b.v]]) return true;
  // GPC puts the other edge's x at this scanline; the horizontal edge, going up
  // to the right, is on the left below
  return add_crossing(S, h, b, x, y, x, m, h.rb, true);
}

// Two edges with a common range of ranks: nothing, a recorded crossing, or the
// pair is not in general position (true).
template <typename C>
__device__ __forceinline__ bool test_edges(const Pair<C> &P, const TEdge &a, const TEdge &b, int lo, int hi) {
  Smem<C> &S = P.S;
  const double m = P.margin;
  const double ylo = S.sy[lo], yhi = S.sy[hi];
  if (a.by == a.ty) return test_horizontal(P, a, b);
  if (b.by == b.ty) return test_horizontal(P, b, a);
  if (ylo == yhi) return !(fabs(a.at(ylo) - b.at(ylo)) > m);
  if (a.w == b.v || b.w == a.v) {
    // the edges of a local extremum: apart at the next vertex y, and from there on
    const bool low = a.rb == b.rb;
    int k = low ? lo + 1 : hi - 1;
    while (S.sy[k] == (low ? ylo : yhi)) k += low ? 1 : -1;
    const double y1 = S.sy[k], y2 = low ? yhi : ylo;
    const double d1 = a.at(y1) - b.at(y1), d2 = a.at(y2) - b.at(y2);
    // polygons of many vertices have ys a few ulps from an extremum: the bound for
    // these two edges rather than for all
    const double own = P.least + 16.0 * gpc::kEps * fmax(fabs(a.tx - a.bx), fabs(b.tx - b.bx));
    return !(fabs(d1) > own && fabs(d2) > own && (d1 > 0.0) == (d2 > 0.0) && fabs(a.dx - b.dx) > 8.0 * gpc::kEps);
  }
  const double s0 = a.at(ylo) - b.at(ylo), s1 = a.at(yhi) - b.at(yhi);
  if (!(fabs(s0) > m && fabs(s1) > m)) return true;
  if ((s0 > 0.0) == (s1 > 0.0)) return false;
  if (S.rside[S.ring[a.v]] == S.rside[S.ring[b.v]]) return true;  // a polygon that crosses itself
  // GPC takes edges of slopes within an epsilon for parallel (layers that are far
  // taller than wide)
  if (!(fabs(a.dx - b.dx) > 8.0 * gpc::kEps)) return true;
  // the beam of the crossing
  int k0 = lo, k1 = hi;
  double d0 = s0, d1 = s1;
  while (k1 - k0 > 1) {
    const int k = (k0 + k1) / 2;
    const double d = a.at(S.sy[k]) - b.at(S.sy[k]);
    if ((d > 0.0) == (s0 > 0.0)) {
      k0 = k;
      d0 = d;
    } else {
      k1 = k;
      d1 = d;
    }
  }
  if (!(fabs(d0) > m && fabs(d1) > m)) return true;
  // GPC's expressions: st the edge on the left at the beam's lower y
  const double yb = S.sy[k0], yt = S.sy[k1], dy = yt - yb;
  const bool a_left = d0 < 0.0;
  const double axb = a.at(yb), axt = a.at(yt), bxb = b.at(yb), bxt = b.at(yt);
  const double sxb = a_left ? axb : bxb, sxt = a_left ? axt : bxt;
  const double exb = a_left ? bxb : axb, ext = a_left ? bxt : axt;
  const double den = (sxt - sxb) - (ext - exb);
  const double r = (exb - sxb) / den;
  return add_crossing(S, a, b, sxb + r * (sxt - sxb), r * dy + yb, r * dy, m + 4.0 * m * fabs(dy / den), k0, a_left);
}

// Order of a node in GPC's sweep: vertices by their y, crossings after the
// vertex below them by their y in the beam.
template <typename C>
__device__ __forceinline__ uint32_t node_key(const Pair<C> &P, int node) {
  if (!(node & 0x8000)) return (uint32_t)P.S.rank[node] << 12;
  const int c = P.crossing(node);
  return ((uint32_t)P.S.beam[c] << 12) + 1u + ((uint32_t)P.S.ord[c] << P.two) + (node & P.two);
}

// Whether the result lies below a contour's local maximum (node m, next: the node
// that follows it).
template <typename C>
__device__ __forceinline__ bool max_is_outer(const Pair<C> &P, int m, int next) {
  if (m & 0x8000) {
    // one quadrant at a crossing belongs to the result, of a union three, of an
    // exclusive or two: below it goes on along the left edge when they are the
    // lower and the upper one
    const int c = P.crossing(m);
    return P.two ? P.S.out[c] == (P.S.aleft[c] ? 0 : 1) : P.convex;
  }
  const TEdge e1 = edge_of(P, m), e0 = edge_of(P, P.prv(m));
  const bool fwd = next & 0x8000 ? P.S.ce[P.S.rside[P.S.ring[m]]][P.crossing(next)] == m : next == P.nxt(m);
  // the result on the left: below when the boundary comes up the right edge (the
  // one with the smaller slope) and goes down the left one
  return fwd ? e0.dx < e1.dx : e1.dx < e0.dx;
}

// Even-odd test of vertex v against the edges of the rings that `take` accepts
// (all threads; the result on all of them).
template <typename C, typename F>
__device__ __forceinline__ bool inside_rings(const Pair<C> &P, int v, F take) {
  Smem<C> &S = P.S;
  const int rv = S.rank[v];
  const double yv = S.sy[rv], xv = P.x(v);
  int odd = 0;
  for (int e = threadIdx.x; e < P.n; e += C::NT) {
    if (!take(S.ring[e])) continue;
    const int w = P.nxt(e), r1 = S.rank[e], r2 = S.rank[w];
    if ((r1 > rv) != (r2 > rv)) {
      const double x1 = P.x(e), x2 = P.x(w), y1 = S.sy[r1], y2 = S.sy[r2];
      if (xv < x1 + (yv - y1) * (x2 - x1) / (y2 - y1)) odd ^= 1;
    }
  }
  if constexpr (C::NT == 32) {
    return __popc(__ballot_sync(0xffffffffu, odd)) & 1;
  } else {
    return __syncthreads_count(odd) & 1;
  }
}

// Minimum of four values over the block.
template <typename C>
__device__ __forceinline__ void block_min4(Smem<C> &S, double *v) {
  for (int k = 0; k < 4; k++)
    for (int o = 16; o; o >>= 1) {
      const double t = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = t < v[k] ? t : v[k];
    }
  if constexpr (C::NT > 32) {
    if ((threadIdx.x & 31) == 0)
      for (int k = 0; k < 4; k++) S.red[k][threadIdx.x >> 5] = v[k];
    __syncthreads();
    for (int k = 0; k < 4; k++)
      for (int w = 0; w < C::NT / 32; w++) v[k] = S.red[k][w] < v[k] ? S.red[k][w] : v[k];
    __syncthreads();
  }
}

// a[k] = the sum of the values before it, a[n] = the sum of all (all threads; the
// counts are complete after the barrier inside).
template <typename C>
__device__ __forceinline__ void block_offsets(Smem<C> &S, int *a, int n) {
  constexpr int NT = C::NT;
  const int per = (n + NT - 1) / NT, k0 = min(n, (int)threadIdx.x * per), k1 = min(n, k0 + per);
  bsync<NT>();
  int sum = 0;
  for (int k = k0; k < k1; k++) sum += a[k];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if ((threadIdx.x & 31) >= o) incl += t;
  }
  if constexpr (NT > 32) {
    int *part = reinterpret_cast<int *>(S.red);
    if ((threadIdx.x & 31) == 31) part[threadIdx.x >> 5] = incl;
    __syncthreads();
    for (int w = 0; w < (int)(threadIdx.x >> 5); w++) incl += part[w];
  }
  int run = incl - sum;
  for (int k = k0; k < k1; k++) {
    const int t = a[k];
    a[k] = run;
    run += t;
  }
  if (threadIdx.x == NT - 1) a[n] = run;
  bsync<NT>();
}

// Result pools (the overlay's) or one pair's area.
struct Sink {
  int32_t *status;
  int64_t *pair_cstart;
  int32_t *pair_ncont;
  int64_t *cont_vstart;
  int32_t *cont_nverts;
  int32_t *cont_hole;
  double *xy;
  unsigned long long *pool;
  int64_t cap_c, cap_v;
  double *area;
};

enum : int { kTraced = 0, kLeft = 1 };

// Intersects one pair (all NT threads); kLeft when the pair is left to the
// scanbeam clippers (nothing written).  pool_full: the status to record when the
// result pools are too small.
template <typename C>
__device__ int trace_pair(Smem<C> &S, int op, const gpc::PolyView &A, const gpc::PolyView &B, const Sink &O, int64_t pair,
                          int pool_full) {
  constexpr int NT = C::NT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = NT / 32;
  const int na = (int)(A.r1 - A.r0), nb = (int)(B.r1 - B.r0);
  bsync<NT>();  // the previous pair's reads
  if (tid == 0) {
    S.ncross = 0;
    S.best = 0;
    S.rstart[0] = 0;
  }
  bool bad = false;  // this thread found the pair not in general position, or too large
  if (na + nb > kMaxRings) return kLeft;
  // ---- rings whose boxes meet a ring of the other polygon (minimax_test,
  // GPC:1656-1709); the others take no part (a difference keeps the subject's, a
  // union and an exclusive or keep all)
  for (int r = 0; r < na + nb; r++) {
    const gpc::PolyView &p = r < na ? A : B;
    const int64_t g = r < na ? A.r0 + r : B.r0 + (r - na);
    double bb[4] = {gpc::kDblMax, gpc::kDblMax, gpc::kDblMax, gpc::kDblMax};
    for (int64_t v = p.ring_vert[g] + tid; v < p.ring_vert[g + 1]; v += NT) {
      const double x = p.xy[2 * v], y = p.xy[2 * v + 1];
      bb[0] = x < bb[0] ? x : bb[0];
      bb[1] = y < bb[1] ? y : bb[1];
      bb[2] = -x < bb[2] ? -x : bb[2];
      bb[3] = -y < bb[3] ? -y : bb[3];
    }
    block_min4(S, bb);
    if (tid == 0) {
      S.rbb[r][0] = bb[0];
      S.rbb[r][1] = bb[1];
      S.rbb[r][2] = -bb[2];
      S.rbb[r][3] = -bb[3];
    }
  }
  bsync<NT>();
  double most = 0.0, most_x = 0.0, wide = 0.0, ymin = gpc::kDblMax, ymax = -gpc::kDblMax;
  int n = 0, nr = 0;
  for (int r = 0; r < na + nb; r++) {
    bool meets = op == PRT_GPC_UNION || op == PRT_GPC_XOR || (op == PRT_GPC_DIFF && r < na);
    for (int q = r < na ? na : 0; q < (r < na ? na + nb : na); q++)
      meets |= r < na ? gpc::bbox_overlap(S.rbb[r], S.rbb[q]) : gpc::bbox_overlap(S.rbb[q], S.rbb[r]);
    if (!meets) continue;
    const gpc::PolyView &p = r < na ? A : B;
    const int64_t g = r < na ? A.r0 + r : B.r0 + (r - na);
    const int64_t len = p.ring_vert[g + 1] - p.ring_vert[g];
    if (len < 3 || n + len > C::kVerts) return kLeft;  // the same on every thread
    if (tid == 0) {
      S.rside[nr] = r < na ? 0 : 1;
      S.rxy[nr] = p.xy + 2 * p.ring_vert[g];
      S.rstart[nr + 1] = n + (int)len;
      S.hit[nr] = 0;
    }
    ymin = fmin(ymin, S.rbb[r][1]);
    ymax = fmax(ymax, S.rbb[r][3]);
    wide = fmax(wide, S.rbb[r][2] - S.rbb[r][0]);
    most_x = fmax(most_x, fmax(fabs(S.rbb[r][0]), fabs(S.rbb[r][2])));
    for (int k = 0; k < 4; k++) most = fmax(most, fabs(S.rbb[r][k]));
    n += (int)len;
    nr++;
  }
  if (!(most < kMostXY)) return kLeft;  // infinities and NaN too
  bsync<NT>();
  // An edge's x at a y is off by at most u|x| for the last addition and 5u w for the
  // slope, the y difference and their product (u half an epsilon, w the x extent):
  // the distance of two by eps(|x| + 6w).  Above twice that and GPC's own epsilon a
  // computed distance has the sign of the true one, and so it has, and is above the
  // epsilon, at every beam between two such ends.
  Pair<C> P{S, n, gpc::kEps * (2.1 * most_x + 16.0 * wide + 1.1), gpc::kEps * (2.1 * most_x + 1.1),
            op != PRT_GPC_UNION};
  if (n > 0) {
    // ---- vertices, and their ys in order
    for (int r = 0; r < nr; r++) {
      const int v0 = S.rstart[r], v1 = S.rstart[r + 1];
      for (int v = v0 + tid; v < v1; v += NT) {
        const double x = S.rxy[r][2 * (v - v0)], y = S.rxy[r][2 * (v - v0) + 1];
        S.vx[v] = x;
        bad |= !(fabs(x) <= most && fabs(y) <= most) || !y_allowed(y);  // NaN; ys next to 0
        S.sy[v] = y;
        S.ring[v] = (uint8_t)r;
      }
    }
    // by buckets of equal y ranges, and in each by counting: stars and rings spread
    // their ys well enough for a few vertices per bucket, more at the top and bottom
    {
      int *bucket = reinterpret_cast<int *>(S.cx);  // no crossings yet
      const int nbuckets = min(n, 6 * C::kCross - 1);
      const double scale = ymax > ymin ? nbuckets / (ymax - ymin) : 0.0;
      auto bucket_of = [&](double y) { return min(nbuckets - 1, (int)((y - ymin) * scale)); };
      for (int b = tid; b <= nbuckets; b += NT) bucket[b] = 0;
      if (bany<NT>(bad)) return kLeft;
      for (int v = tid; v < n; v += NT) atomicAdd(&bucket[bucket_of(S.sy[v])], 1);
      block_offsets(S, bucket, nbuckets);
      for (int v = tid; v < n; v += NT) S.list[atomicAdd(&bucket[bucket_of(S.sy[v])], 1)] = (uint16_t)v;
      bsync<NT>();
      for (int v = tid; v < n; v += NT) {
        const double x = S.vx[v], y = S.sy[v];
        const int b = bucket_of(y), start = b ? bucket[b - 1] : 0, end = bucket[b];
        int before = 0;
        for (int k = start; k < end; k++) {
          const int w = S.list[k];
          const double yw = S.sy[w];
          if (yw < y) {
            before++;
          } else if (yw == y && w != v) {
            const double d = x - S.vx[w];
            before += d > 0.0;
            bad |= !(fabs(d) > P.margin);
          }
        }
        S.rank[v] = (uint16_t)(start + before);
      }
    }
    // GPC leaves out the middle one of three vertices at one y
    for (int v = tid; v < n; v += NT) {
      const double y = S.sy[v];
      bad |= S.sy[P.nxt(v)] == y && S.sy[P.prv(v)] == y;
    }
    if (bany<NT>(bad)) return kLeft;
    for (int v = tid; v < n; v += NT) S.sy[S.rank[v]] = S.rxy[S.ring[v]][2 * (v - S.rstart[S.ring[v]]) + 1];
    // ---- edges per slab of ranks; slabs twice as large while the list is too long
    int shift = C::kSlabShift - 1, slabs;
    do {
      shift++;
      slabs = (n + (1 << shift) - 1) >> shift;
      bsync<NT>();
      for (int s = tid; s <= slabs; s += NT) S.slab0[s] = 0;
      bsync<NT>();
      for (int v = tid; v < n; v += NT) {
        const int r1 = S.rank[v], r2 = S.rank[P.nxt(v)];
        const int lo = min(r1, r2) >> shift, hi = (max(r1, r2) - 1) >> shift;
        for (int s = lo; s <= hi; s++) atomicAdd(&S.slab0[s], 1);
      }
      block_offsets(S, S.slab0, slabs);
    } while (S.slab0[slabs] > C::kList);  // n edges at the most in one slab
    // an edge is listed by its vertex, with kLast when its ring's first vertex is next
    for (int v = tid; v < n; v += NT) {
      const int w = P.nxt(v), r1 = S.rank[v], r2 = S.rank[w];
      const int lo = min(r1, r2) >> shift, hi = (max(r1, r2) - 1) >> shift;
      for (int s = lo; s <= hi; s++)
        S.list[atomicAdd(&S.slab0[s], 1)] = (uint16_t)(v | (w == v + 1 ? 0 : kLast));
    }
    bsync<NT>();
    // slab0[s] is now the end of slab s, the start of slab s + 1
    // ---- every two edges with a common rank and x range, at the one that starts
    // later (of two that start at one vertex, the later listed).  A thread per edge
    // goes through its slab's list; what it finds is queued per warp, as a test is
    // ten times as long as a step of the search and one step in ten finds something.
    {
      uint32_t *queue = S.queue[warp];
      int q = 0;
      auto test_queued = [&](int k) {
        const uint32_t vw = queue[k];
        const TEdge a = edge_of(P, (int)(vw >> 16)), b = edge_of(P, (int)(vw & 0xffffu));
        bad |= test_edges(P, a, b, max(a.rb, b.rb), min(a.rt, b.rt));
      };
      for (int v0 = warp * 32; v0 < n && !__any_sync(0xffffffffu, bad); v0 += NT) {
        const int v = v0 + lane;
        int rb = 0, rt = 0, j = 0, len = 0;
        double xlo = 0.0, xhi = 0.0;
        if (v < n) {
          edge_box(P, v, rb, rt, xlo, xhi);
          const int s = rb >> shift;
          j = s ? S.slab0[s - 1] : 0;
          len = S.slab0[s] - j;
        }
        const int steps = __reduce_max_sync(0xffffffffu, len);
        for (int k = 0; k < steps; k++) {
          bool hit = false;
          int w = 0;
          if (k < len) {
            const int l = S.list[j + k];
            w = l & (kLast - 1);
            const int w2 = l & kLast ? S.rstart[S.ring[w]] : w + 1;
            const int r1 = S.rank[w], r2 = S.rank[w2], bot = min(r1, r2);
            if (bot < rt && max(r1, r2) > rb && (bot < rb || (bot == rb && w < v))) {  // else the later starter looks
              const double x1 = P.x(w), x2 = P.x(w2);
              hit = !(x1 > xhi && x2 > xhi) && !(x1 < xlo && x2 < xlo);
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          if (hit) queue[q + __popc(m & ((1u << lane) - 1))] = (uint32_t)v << 16 | (uint32_t)w;
          q += __popc(m);
          if (q >= 32) {
            __syncwarp();
            test_queued(lane);
            q -= 32;
            __syncwarp();
            const uint32_t rest = queue[32 + lane];
            __syncwarp();
            queue[lane] = rest;
            __syncwarp();
          }
        }
      }
      __syncwarp();
      if (lane < q) test_queued(lane);
    }
    if (bany<NT>(bad)) return kLeft;
  }
  // ---- which side of every ring its material is on
  for (int r = 0; r < nr; r++) {
    const int v0 = S.rstart[r], v1 = S.rstart[r + 1];
    // the ring turns left at its lowest vertex when it runs counter-clockwise
    int low = 0x7fffffff, m = 0;
    for (int v = v0 + tid; v < v1; v += NT)
      if (S.rank[v] < low) {
        low = S.rank[v];
        m = v;
      }
    {
      const int best = __reduce_min_sync(0xffffffffu, low);
      m = __reduce_max_sync(0xffffffffu, low == best ? m : -1);
      low = best;
    }
    if constexpr (NT > 32) {
      if (lane == 0) {
        S.red[0][warp] = (double)low;
        S.red[1][warp] = (double)m;
      }
      __syncthreads();
      for (int w = 0; w < kWarps; w++)
        if (S.red[0][w] < (double)low) {
          low = (int)S.red[0][w];
          m = (int)S.red[1][w];
        }
      __syncthreads();
    }
    const TEdge e1 = edge_of(P, m), e0 = edge_of(P, P.prv(m));
    bool left = e1.dx > e0.dx;  // leaves the minimum by its right edge
    // inside an odd number of the polygon's other rings: a hole
    bool many = false;
    for (int q = 0; q < nr; q++) many |= q != r && S.rside[q] == S.rside[r];
    if (many) {
      const int side = S.rside[r];
      left ^= inside_rings(P, m, [&](int q) { return q != r && S.rside[q] == side; });
    }
    // a difference is the intersection with the other polygon's outside
    if (tid == 0) S.mat[r] = left != (op == PRT_GPC_DIFF && S.rside[r] == 1);
  }
  const int nx = n > 0 ? S.ncross : 0;
  bsync<NT>();
  // ---- crossings in sweep order and along both polygons
  for (int c = tid; c < nx; c += NT) {
    const int k = S.beam[c];
    const double rel = S.crel[c];
    int ord = 0, at[2] = {0, 0};
    int ring[2], e[2];
    bool up[2];
    for (int s = 0; s < 2; s++) {
      e[s] = S.ce[s][c];
      ring[s] = S.ring[e[s]];
      up[s] = S.rank[P.nxt(e[s])] > S.rank[e[s]];
      S.hit[ring[s]] = 1;
    }
    for (int d = 0; d < nx; d++) {
      if (d == c) continue;
      const bool below = S.beam[d] < k || (S.beam[d] == k && S.crel[d] < rel);
      if (S.beam[d] == k && !(fabs(S.crel[d] - rel) > (double)S.ctol[c] + (double)S.ctol[d])) bad = true;
      ord += below ? 1 : 0;
      for (int s = 0; s < 2; s++) {
        const int f = S.ce[s][d];
        at[s] += f < e[s] || (f == e[s] && below == up[s]) ? 1 : 0;
      }
    }
    S.ord[c] = (uint16_t)ord;
    for (int s = 0; s < 2; s++) {
      S.pos[s][c] = (uint16_t)at[s];
      S.seq[s][at[s]] = (uint16_t)c;
    }
    // polygon 0's boundary enters polygon 1 here: the boundary of an intersection
    // goes on along polygon 0, else along polygon 1; of a union the other way round
    const bool same = (up[0] == (S.mat[ring[0]] != 0)) == (up[1] == (S.mat[ring[1]] != 0));
    // of an exclusive or along the left edge, up and down, when the quadrant below
    // belongs to the result, else along the right one
    S.out[c] = ((same != (S.aleft[c] != 0)) != (op == PRT_GPC_UNION || op == PRT_GPC_XOR)) ? 0 : 1;
  }
  if (bany<NT>(bad)) return kLeft;
  // the run that starts at each crossing node: its vertices and the node at its end
  const int nodes = nx << P.two;
  if (nodes > C::kCross) return kLeft;
  for (int t = tid; t < nodes; t += NT) {
    const int c = t >> P.two, s = S.out[c], e = S.ce[s][c], r = S.ring[e], p = S.pos[s][c];
    const int len = S.rstart[r + 1] - S.rstart[r];
    const bool fwd = P.two ? (t & 1) == (int)P.up(e) : S.mat[r] != 0;
    int q = fwd ? p + 1 : p - 1;
    bool wrap = q < 0 || q >= nx || S.ring[S.ce[s][S.seq[s][q]]] != r;
    if (wrap) {  // the ring's first or last crossing
      q = p;
      while (fwd ? q > 0 && S.ring[S.ce[s][S.seq[s][q - 1]]] == r : q + 1 < nx && S.ring[S.ce[s][S.seq[s][q + 1]]] == r)
        q += fwd ? -1 : 1;
    }
    const int d = S.seq[s][q], f = S.ce[s][d];
    S.next[t] = (uint16_t)(d << P.two | (P.two && fwd != P.up(f)));
    S.cnt[t] = (uint16_t)((fwd ? f - e : e - f) + (wrap ? len : 0));
    // the polygons' boundaries enter and leave each other in turn
    if (S.out[d] == s) bad = true;
  }
  if (bany<NT>(bad)) return kLeft;
  // ---- contours: cycles of runs, then whole rings inside the other polygon
  if (tid == 0) {
    int at = 0, nc = 0;
    for (int c = 0; c < nodes; c++) S.cyc[c] = 255;
    for (int c = 0; c < nodes && nc < C::kContours && nc < 250; c++) {
      if (S.cyc[c] != 255) continue;
      S.head[nc] = (uint16_t)at;
      for (int d = c; S.cyc[d] == 255; d = S.next[d]) {
        S.cyc[d] = (uint8_t)nc;
        S.runoff[d] = (uint16_t)at;
        at += 1 + S.cnt[d];
      }
      S.len[nc] = (uint16_t)(at - S.head[nc]);
      nc++;
    }
    for (int c = 0; c < nodes; c++)
      bad |= S.cyc[c] == 255;
    S.ncont = nc;
    S.nodes = at;
  }
  if (bany<NT>(bad)) return kLeft;
  int total = S.nodes, nc = S.ncont;
  if (total > C::kList) return kLeft;
  for (int r = 0; r < nr; r++) {
    if (S.hit[r]) continue;
    const int side = S.rside[r];
    const bool wanted = op != PRT_GPC_UNION && (op != PRT_GPC_DIFF || side == 1);  // inside, else outside
    const bool inside = inside_rings(P, S.rstart[r], [&](int q) { return S.rside[q] != side; });
    if (!P.two && inside != wanted) continue;
    const int len = S.rstart[r + 1] - S.rstart[r];
    if (nc >= C::kContours || total + len > C::kList) return kLeft;
    if (tid == 0) {
      S.head[nc] = (uint16_t)total;
      S.len[nc] = (uint16_t)len;
    }
    const bool fwd = (S.mat[r] != 0) != (P.two && inside);
    for (int k = tid; k < len; k += NT)
      S.list[total + k] = (uint16_t)(fwd ? S.rstart[r] + k : S.rstart[r + 1] - 1 - k);
    total += len;
    nc++;
  }
  for (int t = warp; t < nodes; t += kWarps) {
    const int c = t >> P.two, s = S.out[c], e = S.ce[s][c], r = S.ring[e], r0 = S.rstart[r], r1 = S.rstart[r + 1];
    const int at = S.runoff[t], m = S.cnt[t];
    if (lane == 0) S.list[at] = (uint16_t)(0x8000 | t);
    if (P.two ? (t & 1) == (int)P.up(e) : S.mat[r] != 0) {
      for (int k = lane; k < m; k += 32) {
        const int v = e + 1 + k;
        S.list[at + 1 + k] = (uint16_t)(v < r1 ? v : v - (r1 - r0));
      }
    } else {
      for (int k = lane; k < m; k += 32) {
        const int v = e - k;
        S.list[at + 1 + k] = (uint16_t)(v >= r0 ? v : v + (r1 - r0));
      }
    }
  }
  bsync<NT>();
  // ---- the highest node of every contour, its kind, and for several contours
  // the minimum that each is listed by (one warp per contour)
  if (nc == 1) {  // the usual case, all threads on it
    uint32_t best = 0, at = 0;
    for (int k = tid; k < S.len[0]; k += NT) {
      const uint32_t key = node_key(P, S.list[k]);
      if (key >= best) {
        best = key;
        at = k;
      }
    }
    const uint32_t most_key = __reduce_max_sync(0xffffffffu, best);
    at = __reduce_max_sync(0xffffffffu, best == most_key ? at : 0u);
    if (lane == 0) atomicMax(&S.best, (unsigned long long)most_key << 32 | at);
    bsync<NT>();
    if (tid == 0) {
      S.top[0] = (uint16_t)S.best;
      S.hole[0] = !max_is_outer(P, S.list[S.top[0]], S.list[S.top[0] + 1 < S.len[0] ? S.top[0] + 1 : 0]);
      S.rep[0] = 0;
    }
  }
  for (int c = warp; c < nc && nc > 1; c += kWarps) {
    const int h = S.head[c], m = S.len[c];
    uint32_t best = 0;
    for (int k = lane; k < m; k += 32) best = max(best, node_key(P, S.list[h + k]));
    best = __reduce_max_sync(0xffffffffu, best);
    int at = 0;
    for (int k = lane; k < m; k += 32)
      if (node_key(P, S.list[h + k]) == best) at = k;
    at = __reduce_max_sync(0xffffffffu, at);
    const bool outer = max_is_outer(P, S.list[h + at], S.list[h + (at + 1 < m ? at + 1 : 0)]);
    uint32_t rep = 0;
    // the part of the cycle between two maxima that holds the minimum: at the
    // highest maximum inside it the side that survives the join
    int lo = 1, hi = m - 1;  // offsets from the highest node
    auto node = [&](int o) { return (int)S.list[h + (at + o < m ? at + o : at + o - m)]; };
    for (;;) {
      uint32_t bk = 0;
      uint32_t low = 0xffffffffu;
      for (int o = lo + lane; o <= hi; o += 32) {
        const uint32_t k = node_key(P, node(o));
        low = min(low, k);
        if (o > lo && o < hi && k > node_key(P, node(o - 1)) && k > node_key(P, node(o + 1))) bk = max(bk, k);
      }
      bk = __reduce_max_sync(0xffffffffu, bk);
      if (bk == 0) {
        rep = __reduce_min_sync(0xffffffffu, low);
        break;
      }
      int q = 0;
      for (int o = lo + lane; o <= hi; o += 32)
        if (node_key(P, node(o)) == bk) q = o;
      q = __reduce_max_sync(0xffffffffu, q);
      if (max_is_outer(P, node(q), node(q + 1))) hi = q - 1;
      else lo = q + 1;
    }
    if (lane == 0) {
      S.top[c] = (uint16_t)at;
      S.hole[c] = !outer;
      S.rep[c] = rep;
    }
  }
  bsync<NT>();
  // ---- contours newest minimum first
  for (int c = tid; c < nc; c += NT) {
    int before = 0, off = 0;
    for (int d = 0; d < nc; d++)
      if (S.rep[d] > S.rep[c]) {
        before++;
        off += S.len[d];
      }
    S.place[before] = (uint16_t)c;
    S.off[c] = (uint16_t)off;
  }
  bsync<NT>();
  if (O.area) {
    // shoelace about the first vertex written
    double sum = 0.0;
    for (int p = 0; p < nc; p++) {
      const int c = S.place[p];
      const int h = S.head[c], m = S.len[c];
      auto node = [&](int w) {
        const int o = S.top[c] + (S.hole[c] ? m - w : m - 1 - w);
        return (int)S.list[h + o % m];
      };
      auto px = [&](int v) { return v & 0x8000 ? S.cx[P.crossing(v)] : P.x(v); };
      auto py = [&](int v) { return v & 0x8000 ? S.cy[P.crossing(v)] : P.y(v); };
      const double x0 = px(node(0)), y0 = py(node(0));
      double a = 0.0;
      for (int w = tid; w < m; w += NT) {
        const int u = node(w), v = node(w + 1 < m ? w + 1 : 0);
        a += (px(u) - x0) * (py(v) - y0) - (px(v) - x0) * (py(u) - y0);
      }
      for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if constexpr (NT > 32) {
        if (lane == 0) S.red[0][warp] = a;
        __syncthreads();
        a = 0.0;
        for (int w = 0; w < kWarps; w++) a += S.red[0][w];
        __syncthreads();
      }
      a = 0.5 * fabs(a);
      sum += S.hole[c] ? -a : a;
    }
    if (tid == 0) {
      O.area[pair] = sum;
      O.status[pair] = 0;
    }
    return kTraced;
  }
  // ---- room in the pools
  if (tid == 0) {
    int64_t cb = 0, vb = 0;
    if (nc) {
      cb = (int64_t)atomicAdd(&O.pool[0], (unsigned long long)nc);
      vb = (int64_t)atomicAdd(&O.pool[1], (unsigned long long)total);
    }
    if (cb + nc > O.cap_c || vb + total > O.cap_v) {
      O.pair_ncont[pair] = nc;
      O.pair_cstart[pair] = total;
      O.status[pair] = pool_full;
      bad = true;
    } else {
      O.pair_ncont[pair] = nc;
      O.pair_cstart[pair] = cb;
      O.status[pair] = 0;
    }
    S.cbase = cb;
    S.vbase = vb;
  }
  if (bany<NT>(bad)) return kTraced;
  for (int p = 0; p < nc; p++) {
    const int c = S.place[p];
    const int h = S.head[c], m = S.len[c], t = S.top[c];
    const int64_t v0 = S.vbase + S.off[c];
    if (tid == 0) {
      const int64_t o = S.cbase + p;
      O.cont_nverts[o] = m;
      O.cont_hole[o] = S.hole[c];
      O.cont_vstart[o] = v0;
    }
    for (int w = tid; w < m; w += NT) {
      int o = t + (S.hole[c] ? m - w : m - 1 - w);
      if (o >= m) o -= m;
      const int v = S.list[h + o];
      double2 q;
      q.x = v & 0x8000 ? S.cx[P.crossing(v)] : P.x(v);
      q.y = v & 0x8000 ? S.cy[P.crossing(v)] : P.y(v);
      reinterpret_cast<double2 *>(O.xy)[v0 + w] = q;
    }
  }
  return kTraced;
}

// Pairs of up to 128 vertices in all (1,024; 4,160: one polygon of the 4,096 that
// the uneven layers go up to with a small one; 8,448: two of them).
template <int kTwo>
using Class0 = Class<32, 128, 64, 3, 352, 20, kTwo>;
template <int kTwo>
using Class1 = Class<128, 1024, 256, 3, 3 * 1024, 4, kTwo>;
template <int kTwo>
using Class2 = Class<256, 4160, 256, 3, 4160 * 13 / 8, 2, kTwo>;
template <int kTwo>
using Class3 = Class<512, 8448, 512, 3, 8448 * 3 / 2, 1, kTwo>;
constexpr int kClasses = 4;

}  // namespace trace
}  // namespace prt
