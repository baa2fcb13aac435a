// mv_clip.cu -- the clip kernel of the staged pipeline: ConvexCell::build
// (convex_cell.rs:294-453) over the sorted candidate lists of the shell kernels.
//
// A clip of one cell is a handful of small steps (about four vertices go, six come), so a
// whole warp per cell spends most of its instructions on work that is uniform over the
// warp.  Here a group of 8 lanes builds a cell and a warp builds four cells in lockstep:
// every step below is executed once for all of the warp's cells, with the cells that do
// not take part masked off.  The groups first advance to their next candidate that may
// remove a vertex, two candidates at a time, then clip together.
//
// Per cell in shared memory: the clipping planes (normal, offset), the vertices in the
// reference's order (f32 offset from the generator and the dual planes in filtered mode,
// the f64 location in FP64 mode), the ring's tables and a window of upcoming candidates.
// In filtered mode a vertex's f64 location is recomputed from its dual planes, with the
// operations that created it, where a test is undecided in f32 and when the finished cell
// is written.
//
// What bounds it: instruction latency at 16 warps per SM (the cells' shared memory), and
// instruction fetch: the loop's code has to stay within the 32 KB first-level instruction
// cache, so what is rarely needed is kept out of line and loops are not unrolled.
// 128^3 Poisson cells: with one warp per cell (28 warps per SM, 15.2 k warp-instructions
// per cell) 34.1 ms, in this form (6.9 k) 20.3 ms; replacing a warp's finished cells one by
// one instead of all four together (fuller warps, but the once-per-cell code runs four
// times as often) 36 ms.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdint>

#include "mv_cell_common.cuh"

namespace mv {

#ifndef MV_CLIP_WARPS
#define MV_CLIP_WARPS 2
#endif
#ifndef MV_CLIP_PMAX
#define MV_CLIP_PMAX 37
#endif
#ifndef MV_CLIP_VMAX
#define MV_CLIP_VMAX 48
#endif
#ifndef MV_CLIP_MINB
#define MV_CLIP_MINB 8
#endif

// Capacities of one cell: PMAX planes and VMAX vertices; a cell that outgrows them goes
// on to the next round.
template <int VMAX_, int PMAX_, int WARPS_, int MINB_>
struct ClipTier {
  static constexpr int G = 8;           // lanes per cell
  static constexpr int NG = 32 / G;     // cells per warp
  static constexpr int VMAX = VMAX_;
  static constexpr int PMAX = PMAX_;
  static constexpr int WARPS = WARPS_;
  static constexpr int MINB = MINB_;    // resident blocks per SM the registers are sized for
  static constexpr int WIN = 2 * G;     // candidates in the window (refilled G at a time)
  static constexpr int RMAX = 32;       // removed vertices, ring edges
  static constexpr int NC = VMAX_ / G;  // vertices per lane
  // bytes per plane: words, and the successor of a node outside the ring.  No plane has the
  // number PMAX, so its byte is free: it stays NONE, and a walk that leaves a broken ring
  // goes on inside the table
  static constexpr int PW = (PMAX_ + 4) / 4;
  static constexpr unsigned NONE = PMAX_;
  static constexpr uint32_t NONE4 = 0x01010101u * NONE;
  static_assert(VMAX_ % (2 * G) == 0 && VMAX_ <= 64 && PMAX_ < 255, "tier");
};
using ClipFirst = ClipTier<MV_CLIP_VMAX, MV_CLIP_PMAX, MV_CLIP_WARPS, MV_CLIP_MINB>;
using ClipWide = ClipTier<64, 64, MV_CLIP_WARPS, 6>;

__device__ __forceinline__ uint32_t pack_dual(int i, int j, int k) {
  return (uint32_t)i | ((uint32_t)j << 8) | ((uint32_t)k << 16);
}

// Squared distance of a vertex location to the generator (Vertex::from_dual,
// convex_cell.rs:38-42).
__device__ __forceinline__ double radius2(D3 l, D3 x, int dim) {
  const D3 r = sub(x, D3{l.x, dim >= 2 ? l.y : 0.0, dim == 3 ? l.z : 0.0});
  return dot(r, r);
}

// State shared by both precisions.
template <class T>
struct GroupPlanes {
  double2 pxy[T::PMAX + 1], pzd[T::PMAX + 1];  // plane normals and offsets d = n.p
  double2 wxy[T::WIN], wzd[T::WIN];            // window: half-spaces (HalfSpace::new)
  float2 wc[T::WIN];   // window: f32 bound of the filter without its A term, |x - ngb| rounded up
  uint32_t rd[T::RMAX];  // duals of the removed vertices, in the reference's order
  // byte per plane: the removed triangles that hold it (zero between uses), and its
  // successor (NONE between uses) and predecessor on the ring
  uint32_t plm[T::PW], ring[T::PW], back[T::PW];
  uint16_t pidx[T::PMAX + 1];  // candidate of each bisector plane
  __device__ __forceinline__ D3 normal(int k) const { return {pxy[k].x, pxy[k].y, pzd[k].x}; }
  __device__ __forceinline__ double d(int k) const { return pzd[k].y; }
  // intersect_planes (geometry.rs:68-76) of the dual planes, out of the hot loop's code
  struct Meet {
    D3 loc;
    bool ok;
  };
  __device__ __noinline__ Meet intersect(uint32_t dual) const {
    const int i = dual & 0xff, j = (dual >> 8) & 0xff, k = (dual >> 16) & 0xff;
    Meet m = {{0.0, 0.0, 0.0}, false};
    m.ok = intersect3(normal(i), d(i), normal(j), d(j), normal(k), d(k), &m.loc);
    return m;
  }
  __device__ __noinline__ D3 intersect_loc(uint32_t dual) const {
    D3 l = {0.0, 0.0, 0.0};
    intersect_fast(dual, &l);
    return l;
  }
  // the same, by one reciprocal where the operands allow it
  __device__ __forceinline__ bool intersect_fast(uint32_t dual, D3* loc) const {
    const int i = dual & 0xff, j = (dual >> 8) & 0xff, k = (dual >> 16) & 0xff;
    double det;
    const D3 s = intersect3_parts(normal(i), d(i), normal(j), d(j), normal(k), d(k), &det);
    if (quotients(s, det, loc)) return true;
    const Meet m = intersect(dual);
    *loc = m.loc;
    return m.ok;
  }
};

template <class T>
struct alignas(16) GroupFiltered : GroupPlanes<T> {
  float4 v[T::VMAX];    // f32 offset v - x, dual planes (bytes)
  float4 wf[T::WIN];    // window: e = x - ngb in f32, |e|^2 / 2
  __device__ __forceinline__ uint32_t dual(int q) const { return __float_as_uint(v[q].w); }
  __device__ __forceinline__ void set(int q, D3 loc, D3 x, uint32_t du) {
    v[q] = make_float4(__double2float_rn(loc.x - x.x), __double2float_rn(loc.y - x.y),
                       __double2float_rn(loc.z - x.z), __uint_as_float(du));
  }
  // squared radius of the vertex at position q (Vertex::from_dual)
  __device__ __forceinline__ float radius2_f32(int q, D3, int dim) const {
    const float4 p = v[q];
    const float y = dim >= 2 ? p.y : 0.f, z = dim == 3 ? p.z : 0.f;
    return fmaf(z, z, fmaf(y, y, p.x * p.x));
  }
  // positions from nv on hold the generator itself, which no candidate removes
  __device__ __forceinline__ void set_none(int q, D3) { v[q] = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ D3 loc(int q) const { return this->intersect_loc(dual(q)); }
  __device__ __forceinline__ void move(int to, int from) { v[to] = v[from]; }
};

template <class T>
struct alignas(16) GroupF64 : GroupPlanes<T> {
  double vx[T::VMAX], vy[T::VMAX], vz[T::VMAX];
  double werr[T::WIN];  // window: error bound of the half-space
  uint32_t vd[T::VMAX];
  __device__ __forceinline__ uint32_t dual(int q) const { return vd[q]; }
  __device__ __forceinline__ void set(int q, D3 l, D3, uint32_t du) {
    vx[q] = l.x, vy[q] = l.y, vz[q] = l.z, vd[q] = du;
  }
  __device__ __forceinline__ float radius2_f32(int q, D3 x, int dim) const {
    return __double2float_rn(radius2(D3{vx[q], vy[q], vz[q]}, x, dim));
  }
  __device__ __forceinline__ void set_none(int q, D3 x) { set(q, x, x, 0u); }
  __device__ __forceinline__ D3 loc(int q) const { return {vx[q], vy[q], vz[q]}; }
  __device__ __forceinline__ void move(int to, int from) {
    vx[to] = vx[from], vy[to] = vy[from], vz[to] = vz[from], vd[to] = vd[from];
  }
};

// Padded so that consecutive cells start at different banks.
template <class Base, int PAD = (int)((32 + 16 - sizeof(Base) % 32) % 32)>
struct Padded : Base {
  uint8_t pad[PAD];
};
template <class Base>
struct Padded<Base, 0> : Base {};

template <class T, int PREC>
struct CellOf {
  using type = Padded<GroupFiltered<T>>;
};
template <class T>
struct CellOf<T, MV_PRECISION_FP64> {
  using type = Padded<GroupF64<T>>;
};

// Location of candidate list entry pk (sorted position * 27 + shift code), shifted as
// the reference shifts it (rtree_nn.rs:27-33).
__device__ __forceinline__ D3 cand_loc(const Job& J, uint32_t pk) {
  const int cp = (int)(pk / 27u);
  const int code = (int)(pk - (uint32_t)cp * 27u);
  D3 g = {__ldg(J.sx + cp), __ldg(J.sy + cp), __ldg(J.sz + cp)};
  if (code != 13) g = add(g, D3{J.shift[code][0], J.shift[code][1], J.shift[code][2]});
  return g;
}

// HalfSpace::right_loc (half_space.rs:53-65) of plane k.
template <class SM>
__device__ D3 group_right_loc(const Job& J, const SM& S, const uint32_t* list, int k, D3 x) {
  if (k >= 6) return cand_loc(J, __ldg(list + S.pidx[k]));
  const D3 pr = plane_project(S.normal(k), D3{J.bp[k][0], J.bp[k][1], J.bp[k][2]}, x);
  return sub(scale(2.0, pr), x);
}

// Whether the exact decision (convex_cell.rs:370-382) of a vertex inside the f64 band is
// the zero determinant of five corners of one axis-aligned box (box_corners): the vertex
// is then kept.
template <class SM>
__device__ __noinline__ bool group_box_zero(const Job& J, const SM& S, const uint32_t* list, uint32_t dual,
                                            D3 x, D3 ngb) {
  int64_t A[3], B[3], C[3], Dd[3], W[3];
  iloc(J, x, A);
  iloc(J, group_right_loc(J, S, list, dual & 0xff, x), B);
  iloc(J, group_right_loc(J, S, list, (dual >> 8) & 0xff, x), C);
  iloc(J, group_right_loc(J, S, list, (dual >> 16) & 0xff, x), Dd);
  iloc(J, ngb, W);
  return box_corners(A, B, C, Dd, W);
}

// Largest of a non-negative value over the lanes of each group; called by the whole warp.
template <int G>
__device__ __forceinline__ double group_max(double m) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const double v = __shfl_xor_sync(FULL, m, o);
    m = v > m ? v : m;
  }
  return m;
}

// Squared radii from here on are within f32 rounding of their f64 values (below, the
// squares of the coordinates lose bits or vanish: cells smaller than 1e-15).
constexpr float SQUARE_MIN = 1e-30f;

// The safety radius (convex_cell.rs:443-453) of a group's nv vertices in f64, given their
// largest squared radius in f32: only the vertices within f32 rounding of it can be the
// farthest.
template <int G, class SM>
__device__ __noinline__ double exact_radius(const SM& S, int gl, int nv, float m2, D3 x, int dim) {
  const float least = m2 >= SQUARE_MIN ? m2 * 0.999998f : 0.f;
  double m = 0.0;
#pragma unroll 1
  for (int q = gl; q < nv; q += G) {
    if (S.radius2_f32(q, x, dim) < least) continue;
    const double r2 = radius2(S.loc(q), x, dim);
    m = r2 > m ? r2 : m;
  }
  return 2.0 * sqrt(group_max<G>(m));
}

// Candidate k of a group (`near`) whose f32 distance leaves open whether it is within the
// safety radius, or the list's end: the cell's result when this ends it, -1 when the
// candidate is to be clipped.  su_hi bounds the safety radius.  Called by the whole warp.
template <int G, class SM>
__device__ __noinline__ int at_radius(const Job& J, const StageJob& SJ, const SM& S, const uint32_t* list, int gl,
                                      int item, int info, bool near, int k, int nv, float su_hi, float m2,
                                      D3 x, int dim) {
  const int ncand = info & 0x3fffffff;
  const bool exhausted = (info >> 30) & 1;
  const double rad = near && k == ncand ? SJ.rad[item] : 0.0;
  int got = -1;
  if (near && k == ncand && (exhausted || (double)su_hi < rad * (1.0 - 1e-6))) {
    got = CELL_DONE;  // the whole stream was consumed, or the list reaches beyond the radius
    near = false;
  }
  if (__any_sync(FULL, near)) {
    const double sr = exact_radius<G>(S, gl, near ? nv : 0, m2, x, dim);
    if (near) {
      if (k == ncand) {
        // the list ends: the shell was complete up to its radius (as the fused kernel's shell
        // loop decides); otherwise a later round continues the stream
        got = sr < rad * (1.0 - 1e-12) ? CELL_DONE : CELL_RETRY;
      } else {
        const D3 dx = sub(x, cand_loc(J, __ldg(list + k)));
        const double dist = sqrt(dot(dx, dx));
        if (!(dist > 0.0 && dist <= DBL_MAX))
          got = CELL_ERROR;
        else if (sr < dist)
          got = CELL_DONE;
      }
    }
  }
  return got;
}

// Vertex::from_dual (convex_cell.rs:28-48) at position q.  Returns false when the planes do not meet in a point.
template <class SM>
__device__ __forceinline__ bool add_vertex(SM& S, int q, uint32_t du, D3 x) {
  D3 loc = {0.0, 0.0, 0.0};
  const bool ok = S.intersect_fast(du, &loc);
  S.set(q, loc, x, du);
  return ok;
}

// Window entry sl: candidate c of the list (`in`), or the entry after the last one.
// Filtered: s = e.a + |e|^2 / 2 is certified by T = |e| (cx + C2 |e|) + C1 |e| A with
// A >= |v - x| over the cell's vertices: the bound of setup_batch (mv_cells.cu) with
// |e|_1 <= 1.7321 |e|, its terms gathered by powers of |e| and rounded up.  cx =
// filter_base(x) holds those of the generator alone; an infinite bound leaves the test to
// f64.
constexpr float C1 = 3.0e-7f;    // >= 5.02 2^-24 + 11 2^-53
constexpr float C2 = 2.4031e-7f;  // >= 4.03 2^-24 + 1.7321 (1.0012e-13 + 11 2^-53)
__device__ __forceinline__ float filter_base(D3 x) {
  const double x1 = fabs(x.x) + fabs(x.y) + fabs(x.z);
  return x1 <= 1e15 ? __double2float_ru(1.0001e-13 * (1.0 + 1.002 * x1) + 1.6e-15 * x1) : INFINITY;
}
static __device__ __noinline__ D3 plain_normal(D3 dx, double dist) { return divs(dx, dist); }
template <int PREC, class SM>
__device__ __forceinline__ void fill_window(const Job& J, SM& S, const uint32_t* list, int c, int sl, bool in,
                                            D3 x, float cx) {
  if (!in) {
    S.wc[sl] = make_float2(INFINITY, INFINITY);
    return;
  }
  // location and offset as the reference computes them (convex_cell.rs:333-342)
  const D3 g = cand_loc(J, __ldg(list + c));
  const D3 dx = sub(x, g);
  const double dist = sqrt(dot(dx, dx));
  const float d32 = dist > 0.0 && dist <= DBL_MAX ? __double2float_ru(dist) : INFINITY;
  // HalfSpace::new (half_space.rs:24-34)
  D3 n;
  if (!quotients(dx, dist, &n)) n = plain_normal(dx, dist);
  const D3 p = scale(0.5, add(x, g));
  S.wxy[sl] = make_double2(n.x, n.y);
  S.wzd[sl] = make_double2(n.z, dot(n, p));
  if constexpr (PREC == MV_PRECISION_FILTERED) {
    const bool filt = dist >= 1e-15 && dist <= 1e15;
    const float ex = __double2float_rn(dx.x), ey = __double2float_rn(dx.y), ez = __double2float_rn(dx.z);
    S.wf[sl] = make_float4(ex, ey, ez, 0.5f * fmaf(ez, ez, fmaf(ey, ey, ex * ex)));
    S.wc[sl] = make_float2(filt ? __fmul_ru(d32, __fmaf_ru(C2, d32, cx)) : INFINITY, d32);
  } else {
    S.werr[sl] = 1e-13 * (1.0 + dot(vabs(n), vabs(p)));
    S.wc[sl] = make_float2(0.f, d32);
  }
}

// The swap-remove loop (convex_cell.rs:365-390) of the r removed vertices, one per lane,
// with rm their positions and kr the kept ones in bit-reversed order: removed vertex j at
// position p is replaced by the j-th kept vertex from the end (position q) when
// p < nvf = nv - r, and ends behind the kept ones at the place its swap (or, past nvf,
// the swap of its successor) gives it; from: the kept vertex that the swap before j's
// moved.
template <class SM>
__device__ __forceinline__ void swap_one(SM& S, int j, int r, int nvf, int p, int q, int from) {
  if (j < r) {
    const uint32_t du = S.dual(p);
    if (p < nvf) S.move(p, q);
    S.rd[(p <= nvf ? from : p) - 1 - nvf] = du;
  }
}

// At most 32 vertices and a removed one per lane.
template <class T, class SM>
__device__ __forceinline__ void swap_remove(SM& S, int gl, int r, int rmax, int nv, unsigned rm) {
  unsigned a = rm, b = __brev((nv >= 32 ? FULL : (1u << nv) - 1u) & ~rm);
#pragma unroll 1
  for (int s = 1; s < rmax; s++)
    if (s <= gl) a &= a - 1, b &= b - 1;
  const int q = 31 - (__ffs((int)b) - 1);
  int from = __shfl_up_sync(FULL, q, 1, T::G);
  if (gl == 0) from = nv;
  swap_one(S, gl, r, nv - r, __ffs((int)a) - 1, q, from);
}

// Any number, out of the hot loop's code.
template <class T, class SM>
__device__ __noinline__ void swap_remove_any(SM& S, int gl, int r, int rmax, int nv, unsigned lo, unsigned hi) {
  unsigned long long a = ((unsigned long long)hi << 32) | lo;
  unsigned long long b = __brevll((nv >= 64 ? ~0ull : (1ull << nv) - 1ull) & ~a);
  int last = nv;
  // lane gl takes the removed vertices gl, gl + G, ..
  for (int s = 0; s < gl; s++) a &= a - 1, b &= b - 1;
#pragma unroll 1
  for (int j0 = 0; j0 < rmax; j0 += T::G) {
    const int q = 63 - (__ffsll((long long)b) - 1);
    int from = __shfl_up_sync(FULL, q, 1, T::G);
    if (gl == 0) from = last;
    last = __shfl_sync(FULL, q, T::G - 1, T::G);
    swap_one(S, j0 + gl, r, nv - r, __ffsll((long long)a) - 1, q, from);
#pragma unroll 1
    for (int s = 0; s < T::G; s++) a &= a - 1, b &= b - 1;
  }
}

// The vertices (chunks `open` of this lane) that the filter left open against candidate k,
// whose half-space is plane np: returns the chunks of those removed (bits 0-15), the number
// of box-corner tests (from bit 16), and bit 31 when one needs the multi-limb predicate.
template <class T, int PREC, bool BOX, class SM>
__device__ __noinline__ unsigned undecided(const Job& J, const SM& S, const uint32_t* list, int gl, int np,
                                           int k, unsigned open, D3 x) {
  const D3 n = S.normal(np);
  const double d = S.d(np);
  const D3 g = cand_loc(J, __ldg(list + k));
  const double errb = 1e-13 * (1.0 + dot(vabs(n), vabs(scale(0.5, add(x, g)))));
  unsigned out = 0u;
#pragma unroll 1
  for (unsigned m = open; m; m &= m - 1u) {
    const int c = __ffs(m) - 1, q = c * T::G + gl;
    bool band = true;
    if (PREC == MV_PRECISION_FILTERED) {
      const double s = dot(n, S.loc(q)) - d;
      band = fabs(s) < errb;
      if (!band && s < 0.0) out |= 1u << c;
    }
    if (band) {
      if constexpr (BOX) {
        if (!group_box_zero(J, S, list, S.dual(q), x, g)) out |= 1u << 31;
        out += 1u << 16;
      } else {
        out |= 1u << 31;
      }
    }
  }
  return out;
}

// The node at which the ring of a removed region starts when its first triangle's first
// node is interior: the reference joins the triangles one by one, each time the first (in
// an order that its swaps change) that extends the cycle, and moves the start to the node
// before it in the triangle that closes its fan.  Triangle gl: nodes du, M and N as in the
// clip kernel (N zero in groups that do not take part).  Called by the whole warp.  The cycle holds the reversed edge a of a waiting triangle when N_a meets the
// joined lanes A, and its node a when M_a does.
__device__ __noinline__ int ring_start(uint32_t du, uint32_t M, uint32_t N, int gl, int gbase, int start) {
  uint32_t A = 0x010101u;  // in all three bytes
  int at = gl;             // the lane of the triangle at position gl
  if (gl == 0) N = 0u;     // the first triangle is the cycle
#pragma unroll 1
  for (int i = 1; i < 32; i++) {
    // rotation a of try_extend: the cycle holds the edge t[a+2] -> t[a+1]; t[a] is new (the
    // cycle grows) or follows t[a+1] (t[a+1] becomes interior); flags in bit 7 of byte a
    const uint32_t x = N & A, y = M & A;
    const uint32_t sb = (((x & 0x7f7f7fu) + 0x7f7f7fu) | x) & 0x808080u;
    const uint32_t nb = (((y & 0x7f7f7fu) + 0x7f7f7fu) | y) & 0x808080u;
    const uint32_t can = sb & (~nb | __byte_perm(sb, 0, 0x4102));
    const unsigned all = __ballot_sync(FULL, can != 0u);
    if (all == 0u) break;
    const unsigned bal = (all >> gbase) & 0xffu;
    const uint32_t low = can & (0u - can);
    // t[a], t[a+1], t[a+2] and whether t[a] is in the cycle
    const uint32_t rot = __byte_perm(du, nb & low, low == 0x80u ? 0x4210 : (low == 0x8000u ? 0x5021 : 0x6102));
    // by position, of those not done with
    const unsigned pos = (__ballot_sync(FULL, (bal >> at) & 1u) >> gbase) & 0xffu & (0xffu << i);
    const int found = __ffs(pos) - 1;
    const int src = __shfl_sync(FULL, at, found, 8), head = __shfl_sync(FULL, at, i, 8);
    const uint32_t w = __shfl_sync(FULL, rot, src, 8);
    if (bal != 0u) {
      if (gl == found) at = head;  // swap(i, found): position i is done with
      A |= 0x010101u << src;
      if (gl == src) N = 0u;
      if ((w >> 24) != 0u && start == (int)((w >> 8) & 0xff)) start = w & 0xff;
    }
  }
  return start;
}

// The ring of a group (`on`) that removes more vertices, or gets more edges, than it has
// lanes: compute_boundary + SimpleCycle through shared memory (S.ring: successors; S.rd:
// the removed triangles, which the ring's nodes replace in cycle order).  Called by the
// whole warp.  Returns the number of edges, bit 16 set when the ring's start moved; 0 when
// a triangle cannot be joined.
template <class T, class SM>
__device__ __noinline__ unsigned ring_wide(SM& S, int gl, int gbase, bool on, int r) {
  constexpr int G = T::G;
  constexpr unsigned GM = (1u << G) - 1u;
  uint8_t* const rptr = reinterpret_cast<uint8_t*>(S.ring);
  if (on)
#pragma unroll 1
    for (int i = gl; i < T::PW; i += G) S.ring[i] = T::NONE4;
  __syncwarp();
  const uint32_t d0 = on ? S.rd[0] : 0u;
  int start = d0 & 0xff, E = 3;
  bool moved = false, ok = true;
  const uint32_t nx = __byte_perm(d0, 0, 0x4021);  // t1, t2, t0
  if (on && gl < 3) rptr[(d0 >> (8 * gl)) & 0xff] = (uint8_t)((nx >> (8 * gl)) & 0xff);
  __syncwarp();
#pragma unroll 1
  for (int i = 1;; i++) {
    bool step = on && ok && i < r;
    if (!__any_sync(FULL, step)) break;
    uint32_t head = 0u;  // lane 0: the triangle at position i
#pragma unroll 1
    for (int base = i;; base += G) {
      const int idx = base + gl;
      const uint32_t du = step && idx < r ? S.rd[idx] : 0u;
      const unsigned t0 = du & 0xff, t1 = (du >> 8) & 0xff, t2 = (du >> 16) & 0xff;
      const unsigned p0 = rptr[t0], p1 = rptr[t1], p2 = rptr[t2];
      const bool s0 = p2 == t1, s1 = p0 == t2, s2 = p1 == t0;
      const bool o0 = p0 == T::NONE, o1 = p1 == T::NONE, o2 = p2 == T::NONE;
      const bool x0 = s0 && (o0 || s2), x1 = s1 && (o1 || s0), x2 = s2 && (o2 || s1);
      const bool can = du != 0u && (x0 || x1 || x2);
      const bool grow_l = x0 ? o0 : (x1 ? o1 : o2);
      uint32_t win = __byte_perm(du, grow_l ? 1u : 0u, x0 ? 0x4210 : (x1 ? 0x4021 : 0x4102));
      if (base == i) head = du;
      const unsigned bal = (__ballot_sync(FULL, can) >> gbase) & GM;
      const int src = bal ? __ffs(bal) - 1 : 0;
      win = __shfl_sync(FULL, win, gbase + src);
      const unsigned ta = win & 0xff, tb = (win >> 8) & 0xff, tc = (win >> 16) & 0xff;
      const bool grow = (win >> 24) != 0u, did = step && bal != 0u;
      if (did && gl == 0) {
        rptr[tc] = (uint8_t)ta;
        rptr[grow ? ta : tb] = (uint8_t)(grow ? tb : T::NONE);
        S.rd[base + src] = head;  // swap(i, found): position i is done with
      }
      if (did) E += grow ? 1 : -1;
      if (did && !grow && start == (int)tb) start = ta, moved = true;
      step = step && !did;
      if (step && base + G >= r) ok = step = false;
      __syncwarp();
      if (!__any_sync(FULL, step)) break;
    }
  }
  if (on && ok) {
    if (gl == 0 && E <= T::RMAX) {
      int cur = start;
#pragma unroll 1
      for (int e = 0; e < E; e++) {
        S.rd[e] = (uint32_t)cur;
        cur = rptr[cur];
      }
    }
    __syncwarp(GM << gbase);
#pragma unroll 1
    for (int i = gl; i < T::PW; i += G) S.ring[i] = T::NONE4;
  }
  __syncwarp();
  return ok ? (unsigned)E | (moved ? 1u << 16 : 0u) : 0u;
}

// Writes the finished cells (`on`) of a warp's groups as records (see rec_words), their
// safety radii (convex_cell.rs:443-453) from the vertices' f64 locations; a group's lanes
// share its planes and vertices.  Called by the whole warp; returns false in groups whose
// record does not fit the buffer.
template <class T, class SM>
__device__ __noinline__ bool write_group_record(const Job& J, const StageJob& SJ, const SM& S,
                                                const uint32_t* list, int gl, unsigned gmask, bool on,
                                                int item, D3 x, int np, int nv) {
  constexpr int G = T::G;
  bool onb = SJ.full_records != 0;  // a vertex on a boundary plane
#pragma unroll 1
  for (int q = gl; q < (on ? nv : 0); q += G) {
    const uint32_t du = S.dual(q);
    onb |= (du & 0xff) < 6u || (du & 0xff00) < 0x600u || (du & 0xff0000) < 0x60000u;
  }
  const int pb = (__ballot_sync(FULL, onb) & gmask) ? 0 : 6;
  const int ps = np - pb;
  const int words = (int)rec_words(np, nv, pb);
  unsigned long long off = 0;
  if (gl == 0 && on) off = atomicAdd(SJ.rec_counter, (unsigned long long)words);
  off = __shfl_sync(FULL, off, 0, G);
  const bool fits = on && (int64_t)off + words <= SJ.rec_cap;
  double* R = SJ.rec + off;
#pragma unroll 1
  for (int k = gl; k < (fits ? ps : 0); k += G) {
    const int pl = k + pb;
    const D3 nn = S.normal(pl);
    D3 p;
    int right = -1, code = 13;
    if (pl < 6) {
      p = {J.bp[pl][0], J.bp[pl][1], J.bp[pl][2]};
    } else {
      const uint32_t pk = __ldg(list + S.pidx[pl]);
      p = scale(0.5, add(x, cand_loc(J, pk)));
      const int cp = (int)(pk / 27u);
      right = __ldg(J.sid + cp);
      code = (int)(pk - (uint32_t)cp * 27u);
    }
    rec_plane(R, k, nn, S.d(pl), plane_project(nn, p, x), right, code);  // Plane::project_onto
  }
  double m = 0.0;
  const int dim = J.dim;
#pragma unroll 1
  for (int q = gl; q < (fits ? nv : 0); q += G) {
    const D3 l = S.loc(q);
    rec_vertex(R, ps, q, l, S.dual(q));
    const double r2 = radius2(l, x, dim);
    m = r2 > m ? r2 : m;
  }
  m = group_max<G>(m);
  if (gl == 0 && fits) {
    rec_header(R, np, nv, pb, 2.0 * sqrt(m));
    SJ.rec_off[item] = (int64_t)off;
  }
  return fits;
}

// BOX: band tests that are box-corner zeros are decided here (lattice-like inputs).
template <class T, int PREC, bool MULTI, bool BOX>
__global__ void __launch_bounds__(32 * T::WARPS, T::MINB)
    clip_kernel(const __grid_constant__ Job J0, const __grid_constant__ StageJob SJ,
                const __grid_constant__ JobTable TB) {
  constexpr int G = T::G, NC = T::NC, WIN = T::WIN;
  constexpr bool FILT = PREC == MV_PRECISION_FILTERED;
  constexpr unsigned GM = (1u << G) - 1u;
  using Cell = typename CellOf<T, PREC>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gl = lane & (G - 1), gbase = lane & ~(G - 1);
  const unsigned gmask = GM << gbase;
  Cell& S = reinterpret_cast<Cell*>(smem_raw)[warp * T::NG + lane / G];
  auto gballot = [&](bool p) -> unsigned { return (__ballot_sync(FULL, p) >> gbase) & GM; };
  // event counts of the cells this lane's group finished (lane 0 of the group; undecided
  // and exact tests on every lane)
  unsigned c_ngb = 0, c_pl = 0, c_ring = 0, c_und = 0, c_ex = 0;

  // the group's cell: its item (-1: none), and whether it is still being built
  int item = -1, gpos = 0, jb = 0, self = 0, info = 0, dim = 3, res = CELL_RETRY, err = 0;
  bool act = false;
  D3 x = {0.0, 0.0, 0.0};
  float cx = 0.f;
  int nv = 0, np = 0;
  // next candidate; the window holds candidates [k, wlim), INT_MAX: up to the list's end
  int k = 0, wlim = 0;
  unsigned n_ring = 0, n_und = 0, n_ex = 0;
  // f32 bounds of the safety radius: every vertex is within su_hi / 2 of x; a candidate
  // nearer than su_lo is certainly within the safety radius, one farther than su_hi
  // certainly beyond it.  The f64 value is computed where these leave it open and for the
  // finished cell
  float su_lo = 0.f, su_hi = 0.f, A32 = 0.f, m2 = 0.f;  // m2: the largest squared radius
  auto set_radius = [&](float m) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
    m2 = m;
    float su;  // within 1e-6 of 2 sqrt(m)
    asm("sqrt.approx.f32 %0, %1;" : "=f"(su) : "f"(m));
    su += su;
    // out of the range where su is accurate (a square near the smallest f32 or the largest)
    // the bounds are no numbers, which tells nothing of any candidate: all are compared in f64
    if (!(m >= SQUARE_MIN && m <= 1e37f)) su = NAN;
    su_lo = su * 0.999998f;
    su_hi = su * 1.000002f;
    // |v - x| <= A32 (the extruded dimensions add up to 0.5 each)
    A32 = 0.5000001f * su_hi + (dim == 3 ? 0.f : (dim == 2 ? 0.51f : 0.7212f));
    if (!(A32 <= 1e15f)) A32 = INFINITY;
  };

#pragma unroll 1
  for (;;) {
    // ---- the next cells; inactive ones, and those without a list, are passed by ----
    bool need = lane / G < SJ.per_warp;
    res = CELL_RETRY;
#pragma unroll 1
    for (;;) {
      const unsigned want = __ballot_sync(FULL, need);
      if (want == 0u) break;
      int first = 0;
      if (lane == 0) first = (int)atomicAdd(SJ.work + 1, (unsigned)__popc(want) / G);
      first = __shfl_sync(FULL, first, 0);
      if (need) {
        item = first + __popc(want & ((1u << gbase) - 1u)) / G;
        if (item >= SJ.nitems) {
          item = -1;
        } else {
          gpos = SJ.order != nullptr ? __ldg(SJ.order + SJ.item0 + item) : SJ.item0 + item;
          // the cell's tessellation (batch builds): its Job and its local position
          jb = MULTI ? job_of(TB, gpos) : 0;
          const Job& J = MULTI ? TB.jobs[jb] : J0;
          self = __ldg(J.sid + (MULTI ? gpos - __ldg(TB.pos_base + jb) : gpos));
          info = SJ.info[item];
          if (info > 0) {
            act = true;
            need = false;
          } else {
            const bool masked = J.mask != nullptr && J.mask[self] == 0;
            if (masked && gl < 3) J.centroid[3 * (int64_t)self + gl] = 0.0;  // VoronoiCell::default()
            if (gl == 0) {
              SJ.rec_off[item] = -1;
              if (masked) {
                J.volume[self] = 0.0;
                J.safety_radius[self] = 0.0;
                J.face_count[self] = 0;
                J.stage_off[self] = 0;
              } else {
                const unsigned at = atomicAdd(SJ.retry_count, 1u);
                SJ.retry_list[at] = gpos;
              }
            }
            item = -1;
          }
        }
      }
      if (first + __popc(want) / G >= SJ.nitems) need = false;
    }
    if (!__any_sync(FULL, act)) break;
    // ---- ConvexCell::init (convex_cell.rs:294-312): the cuboid's planes; its vertices are
    // made with the other groups' new ones ----
    if (act) {
      const Job& J = MULTI ? TB.jobs[jb] : J0;
      res = CELL_RETRY, err = 0;
      x = load_gen(J, self);
      dim = J.dim;
      cx = filter_base(x);
      nv = 0, np = 5, k = 0, wlim = 1;
      n_ring = n_und = n_ex = 0u;
#pragma unroll 1
      for (int i = gl; i < 6; i += G) {
        S.pxy[i] = make_double2(J.bn[i][0], J.bn[i][1]);
        S.pzd[i] = make_double2(J.bn[i][2], J.bd[i]);
      }
#pragma unroll 1
      for (int i = gl; i < T::PW; i += G) S.plm[i] = 0u, S.ring[i] = T::NONE4, S.back[i] = 0u;
#pragma unroll 1
      for (int q = gl; q < T::VMAX; q += G) S.set_none(q, x);
    }
    __syncwarp();

    const Job& J = MULTI ? TB.jobs[jb] : J0;
    const uint32_t* const list = SJ.cand + (int64_t)(item < 0 ? 0 : item) * SJ.cstride;
    const int ncand = info & 0x3fffffff;
    // ---- ConvexCell::build (convex_cell.rs:316-356), one clip in every active group at a time ----
    int pass = 0;
#pragma unroll 1
    for (;; pass++) {
      if (!__any_sync(FULL, act)) break;
      asm volatile("" : "+r"(pass));  // one copy of the loop's code: it has to stay in the instruction cache
      const int nvmax = (int)__reduce_max_sync(FULL, act ? (unsigned)nv : 0u);
      // the vertices this pass makes: E of them from position nvf on, lane gl's from planes du
      bool hit = act, wide = false;
      int nvf = 0, E = 8;
      uint32_t du = 0u;
      if (pass == 0) {  // the cuboid's vertices
        int i0 = 0, i1 = 0, i2 = 0;
        cuboid_duals(gl, &i0, &i1, &i2);
        du = pack_dual(i0, i1, i2);
      } else {
      // each group advances to its next candidate that may remove a vertex, two candidates at
      // a time.  vm: the chunks in which this lane has a vertex
      const unsigned vm = nv > gl ? (1u << ((nv - gl + G - 1) / G)) - 1u : 0u;
      bool search = act;
      hit = false;
      const float A1 = C1 * A32;
      while (__any_sync(FULL, search)) {
        float2 cc = S.wc[k & (WIN - 1)], cd = S.wc[(k + 1) & (WIN - 1)];
        if (__any_sync(FULL, search && (k + 2 > wlim || !(cc.y < su_lo)))) {
          if (__any_sync(FULL, search && k + 2 > wlim)) {
            // the next G candidates of every group whose window has room; the entry after the
            // last candidate, like a degenerate one, is out of reach of any safety radius
            const bool fill = act && wlim - k <= WIN - G;
            const int c = wlim + gl;
            if (fill && c <= ncand) fill_window<PREC>(J, S, list, c, c & (WIN - 1), c < ncand, x, cx);
            if (fill) wlim = wlim + G <= ncand ? wlim + G : INT_MAX;
            __syncwarp();
            cc = S.wc[k & (WIN - 1)], cd = S.wc[(k + 1) & (WIN - 1)];
          }
          // the list's end, a degenerate distance, or not certainly within the safety radius
          bool near = search && !(cc.y < su_lo);
          if (near && cc.y > su_hi && cc.y < INFINITY) {  // certainly beyond it (convex_cell.rs:343-345)
            res = CELL_DONE;
            near = search = act = false;
          }
          if (__any_sync(FULL, near)) {
            const int got = at_radius<G>(J, SJ, S, list, gl, item, info, near, k, nv, su_hi, m2, x, dim);
            if (near && got >= 0) {
              res = got;
              if (got == CELL_ERROR) err = MV_ERR_DEGENERATE;  // convex_cell.rs:342
              search = act = false;
            }
          }
        }
        const bool two = cd.y < su_lo;
        bool f0, f1;  // not certain to keep all of this lane's vertices
        if constexpr (FILT) {
          const float4 f = S.wf[k & (WIN - 1)], g = S.wf[(k + 1) & (WIN - 1)];
          float m0 = INFINITY, m1 = INFINITY;
          const float4* v = S.v + gl;
          int left = nvmax;
#pragma unroll 1
          do {
            const float4 p = v[0], q = v[G];  // VMAX is a multiple of 2 G
            const float s0 = fmaf(f.z, p.z, fmaf(f.y, p.y, fmaf(f.x, p.x, f.w)));
            const float s1 = fmaf(g.z, p.z, fmaf(g.y, p.y, fmaf(g.x, p.x, g.w)));
            const float s2 = fmaf(f.z, q.z, fmaf(f.y, q.y, fmaf(f.x, q.x, f.w)));
            const float s3 = fmaf(g.z, q.z, fmaf(g.y, q.y, fmaf(g.x, q.x, g.w)));
            m0 = fminf(m0, fminf(s0, s2));
            m1 = fminf(m1, fminf(s1, s3));
            v += 2 * G;
            left -= 2 * G;
          } while (left > 0);
          f0 = !(m0 > __fmaf_ru(cc.y, A1, cc.x)), f1 = !(m1 > __fmaf_ru(cd.y, A1, cd.x));
        } else {
          const int sl = k & (WIN - 1), sl1 = (k + 1) & (WIN - 1);
          const D3 n0 = {S.wxy[sl].x, S.wxy[sl].y, S.wzd[sl].x}, n1 = {S.wxy[sl1].x, S.wxy[sl1].y, S.wzd[sl1].x};
          const double d0 = S.wzd[sl].y, e0 = S.werr[sl], d1 = S.wzd[sl1].y, e1 = S.werr[sl1];
          f0 = f1 = false;
#pragma unroll 1
          for (int q = gl; q < nvmax + gl; q += G) {
            const D3 l = {S.vx[q], S.vy[q], S.vz[q]};
            f0 |= dot(n0, l) - d0 < e0;
            f1 |= dot(n1, l) - d1 < e1;
          }
        }
        const bool h0 = (__ballot_sync(FULL, f0) & gmask) != 0u;
        const bool h1 = (__ballot_sync(FULL, f1 && two) & gmask) != 0u;
        if (search) {
          hit = h0 || h1;
          k += h0 ? 0 : (two && !h1 ? 2 : 1);
          search = !hit;
        }
      }
      if (!__any_sync(FULL, hit)) continue;

      // bit c of rl / ul: this lane's vertex of chunk c is certainly removed / not certainly kept
      unsigned rl = 0u, ul = 0u;
      {
        const int sl = k & (WIN - 1);
        unsigned bit = 1u;
        if constexpr (FILT) {
          const float4 f = S.wf[sl];
          const float2 cc = S.wc[sl];
          const float T0 = __fmaf_ru(cc.y, A1, cc.x);
#pragma unroll 1
          for (int q = gl; q < nvmax + gl; q += G, bit += bit) {
            const float4 p = S.v[q];
            const float s0 = fmaf(f.z, p.z, fmaf(f.y, p.y, fmaf(f.x, p.x, f.w)));
            if (!(s0 > T0)) ul |= bit;
            if (s0 < -T0) rl |= bit;
          }
        } else {
          const D3 n0 = {S.wxy[sl].x, S.wxy[sl].y, S.wzd[sl].x};
          const double d0 = S.wzd[sl].y, e0 = S.werr[sl];
#pragma unroll 1
          for (int q = gl; q < nvmax + gl; q += G, bit += bit) {
            const double s0 = dot(n0, D3{S.vx[q], S.vy[q], S.vz[q]}) - d0;
            const bool b0 = fabs(s0) < e0;
            if (b0 || s0 < 0.0) ul |= bit;
            if (!b0 && s0 < 0.0) rl |= bit;
          }
        }
        if (!hit) rl = ul = 0u;
        rl &= vm, ul &= vm;
      }

      // ---- candidate k of the groups with a hit: its half-space into the next plane's slot ----
      {
        const int sl = k & (WIN - 1);
        if (hit && gl == 0) S.pxy[np] = S.wxy[sl];
        if (hit && gl == 1) S.pzd[np] = S.wzd[sl];
        if (hit && gl == 2) S.pidx[np] = (uint16_t)k;
      }
      __syncwarp();

      // ---- vertices the f32 test left open take the reference's f64 test; inside the f64
      // band the reference decides with the exact in-sphere predicate (half_space.rs:40-47),
      // a zero determinant keeping the vertex.  Five corners of one axis-aligned box (every
      // band test of a quantised lattice) are such a zero without multi-limb arithmetic
      // (BOX); any other band test sends the cell to the fused kernel ----
      const unsigned open = hit ? ul & ~rl : 0u;
      if (__any_sync(FULL, open != 0u)) {
        bool hard = false;
        if (open) {
          if constexpr (FILT) n_und += __popc(open);
          const unsigned got = undecided<T, PREC, BOX>(J, S, list, gl, np, k, open, x);
          hard = got >> 31;
          n_ex += (got >> 16) & 0x7fffu;
          rl |= got & 0xffffu;
        }
        if ((__ballot_sync(FULL, hard) & gmask) != 0u && hit) {
          res = CELL_EXACT;
          hit = act = false;
        }
        __syncwarp();
      }
      // positions of the removed vertices
      unsigned rm_lo = 0u, rm_hi = 0u;
#pragma unroll
      for (int c = 0; c < 32 / G; c++) rm_lo |= gballot((rl >> c) & 1u) << (c * G);
      if (nvmax > 32) {
#pragma unroll
        for (int c = 32 / G; c < NC; c++) rm_hi |= gballot((rl >> c) & 1u) << (c * G - 32);
      }
      const int r_all = __popc(rm_lo) + __popc(rm_hi);
      if (hit) {
        if (r_all == 0) {
          k++;  // an undecided vertex was kept
          hit = false;
        } else if (np >= T::PMAX || r_all > T::RMAX) {
          res = CELL_OVERFLOW;
          hit = act = false;
        }
      }
      if (!__any_sync(FULL, hit)) continue;

      // ---- swap-remove loop (convex_cell.rs:365-390) as a closed-form permutation: removed
      // vertex j (ascending) below nvf is replaced by the kept vertex j-th from the end, and
      // ends where the reference's swaps leave it; only its dual is needed, in rd ----
      const int r = hit ? r_all : 0;
      nvf = nv - r;
      const int rmax = (int)__reduce_max_sync(FULL, (unsigned)r);
      if (nvmax <= 32 && rmax <= G)
        swap_remove<T>(S, gl, r, rmax, nv, rm_lo);
      else
        swap_remove_any<T>(S, gl, r, rmax, nv, rm_lo, rm_hi);
      __syncwarp();

      // ---- the ring of the removed region: compute_boundary + SimpleCycle
      // (convex_cell.rs:421-441, simple_cycle.rs:17-78), one removed triangle per lane.  M
      // holds, per node of the lane's triangle (byte a: t[a]), the lanes whose triangles have
      // it, N (byte a: the edge t[a+1] t[a+2]) the lane across each edge: the dual of a convex
      // cell is a triangulated sphere, so an edge is in two triangles ----
      uint8_t* const next = reinterpret_cast<uint8_t*>(S.ring);
      uint8_t* const prev = reinterpret_cast<uint8_t*>(S.back);
      int start;
      bool moved;
      {
        const bool mine = hit && gl < r;
        du = mine ? S.rd[gl] : 0u;
        const unsigned t0 = du & 0xff, t1 = (du >> 8) & 0xff, t2 = (du >> 16) & 0xff;
        if (mine) {
          atomicOr(&S.plm[t0 >> 2], 1u << (gl + 8 * (t0 & 3)));
          atomicOr(&S.plm[t1 >> 2], 1u << (gl + 8 * (t1 & 3)));
          atomicOr(&S.plm[t2 >> 2], 1u << (gl + 8 * (t2 & 3)));
        }
        start = __shfl_sync(FULL, du, 0, G) & 0xff;
        __syncwarp();
        uint8_t* const pb = reinterpret_cast<uint8_t*>(S.plm);
        const uint32_t M = mine ? (uint32_t)pb[t0] | ((uint32_t)pb[t1] << 8) | ((uint32_t)pb[t2] << 16) : 0u;
        __syncwarp();
        uint32_t N = __byte_perm(M, 0, 0x4021) & __byte_perm(M, 0, 0x4102) & ~(0x010101u << gl);
        // the ring's edges: those with no removed triangle across
        const bool b0 = mine && !(N & 0xffu), b1 = mine && !(N & 0xff00u), b2 = mine && !(N & 0xff0000u);
        if (b0) next[t1] = (uint8_t)t2, prev[t2] = (uint8_t)t1;
        if (b1) next[t2] = (uint8_t)t0, prev[t0] = (uint8_t)t2;
        if (b2) next[t0] = (uint8_t)t1, prev[t1] = (uint8_t)t0;
        if (mine) pb[t0] = 0, pb[t1] = 0, pb[t2] = 0;
        E = __popc(gballot(b0)) + __popc(gballot(b1)) + __popc(gballot(b2));
        wide = hit && (r > G || E > G);
        __syncwarp();
        // the ring starts at the first triangle's first node; when that becomes interior, at
        // the node before it in the triangle that closed its fan, which takes the reference's
        // order to tell
        moved = hit && !wide && next[start] == T::NONE;
        if (__any_sync(FULL, moved)) {
          if (!moved) N = 0u;
          start = ring_start(du, M, N, gl, gbase, start);
          // a cut that removes every vertex leaves no edge (and no first node on one): what the
          // reference's loop makes of it, a ring of two nodes, only that loop tells
          wide = wide || (moved && E < 3);
        }
      }
      int u, w;
      {
        // the node gl steps along the ring, from its start forwards or backwards
        const bool fwd = 2 * gl <= E;
        const int steps = wide || !hit ? 0 : (fwd ? gl : E - gl);
        const uint8_t* const tab = fwd ? next : prev;
        u = start;
#pragma unroll
        for (int s = 0; s < G / 2; s++)
          if (s < steps) u = tab[u];
        w = next[u];
        // one cycle through the start: each node's successor is the next lane's node
        const int un = __shfl_sync(FULL, u, gl + 1 < E ? gl + 1 : 0, G);
        const bool on = hit && !wide && gl < E;
        const bool bad = on && (w != un || u == (int)T::NONE || (gl > 0 && u == start));
        __syncwarp();
        if (on) next[u] = (uint8_t)T::NONE;
        const unsigned broken = __ballot_sync(FULL, bad) & gmask;
        wide = wide || broken != 0u;
      }
      if (__any_sync(FULL, wide)) {
        // more removed vertices or ring edges than lanes, or a ring that only the reference's
        // own loop decides: the ring through shared memory
        const unsigned got = ring_wide<T>(S, gl, gbase, wide && hit, r);
        if (wide) E = got & 0xffff, moved = got >> 16;
        if (wide && hit && got == 0u) {
          res = CELL_ERROR, err = MV_ERR_RING;
          hit = act = false;
        }
      }
      if (hit && (nvf + E > T::VMAX || E > T::RMAX)) {
        res = CELL_OVERFLOW;
        hit = act = false;
      }
      n_ring += hit && moved;

      // the ring's edges (u, w) in SimpleCycle iteration order, each with the new plane
      du = pack_dual(u, w, np);
      }

      // ---- the new vertices, then update_safety_radius (convex_cell.rs:443-453) ----
      {
        const int emax = (int)__reduce_max_sync(FULL, hit ? (unsigned)E : 0u);
        bool ok = true;
#pragma unroll 1
        for (int e0 = 0; e0 < emax; e0 += G) {
          const int e = e0 + gl;
          if (hit && e < E) {
            if (wide) du = pack_dual((int)S.rd[e], (int)S.rd[e + 1 == E ? 0 : e + 1], np);
            ok &= add_vertex(S, nvf + e, du, x);
          }
        }
        __syncwarp();
        if ((__ballot_sync(FULL, !ok) & gmask) != 0u && hit) {
          res = CELL_ERROR, err = MV_ERR_DET;
          hit = act = false;
        }
      }
      {
        float mk = 0.f;
#pragma unroll 1
        for (int q = gl; q < (hit ? nvf + E : 0); q += G) mk = fmaxf(mk, S.radius2_f32(q, x, dim));
        const float lo = su_lo, hi = su_hi, a = A32, m = m2;
        set_radius(mk);
        if (hit) {
#pragma unroll 1
          for (int q = nvf + E + gl; q < nv; q += G) S.set_none(q, x);
          nv = nvf + E;
          np++;
          k++;
        } else {
          su_lo = lo, su_hi = hi, A32 = a, m2 = m;
        }
      }
      __syncwarp();
    }

    // ---- the finished cells' records for the integral kernel ----
    const bool written =
        write_group_record<T>(J, SJ, S, list, gl, gmask, item >= 0 && res == CELL_DONE, item, x, np, nv);
    if (item >= 0 && res == CELL_DONE) {
      if (written) {
        if (gl == 0) c_ngb += (unsigned)(k - 1), c_pl += (unsigned)(np - 6), c_ring += n_ring;
        c_und += n_und;
        c_ex += n_ex;
      } else {
        res = CELL_RETRY;
      }
    }
    if (gl == 0 && item >= 0 && res != CELL_DONE) {
      SJ.rec_off[item] = -1;
      if (res == CELL_ERROR) {
        atomicCAS(J.status + STATUS_CODE, 0, err);
        atomicMin(J.status + STATUS_CELL, self + J.id_base);
      } else if (res == CELL_EXACT) {
        const unsigned at = atomicAdd(SJ.fused_count, 1u);
        SJ.fused_list[at] = gpos;
      } else {
        const unsigned at = atomicAdd(SJ.retry_count, 1u);
        SJ.retry_list[at] = gpos;
      }
    }
    item = -1;
    __syncwarp();
  }
  const unsigned v[5] = {c_ngb, c_pl, c_ring, c_und, c_ex};
  const int slot[5] = {ST_NEIGHBOURS, ST_PLANES, ST_SERIAL_RING, ST_F32_UNDECIDED, ST_EXACT};
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const unsigned s = __reduce_add_sync(FULL, v[i]);
    if (lane == 0 && s) atomicAdd(J0.stats + slot[i], (unsigned long long)s);
  }
}

// ---------------------------------------------------------------- launchers --
using ClipFn = void (*)(const Job, const StageJob, const JobTable);

template <class T>
static ClipFn clip_fn(int precision, bool multi, bool box) {
  if (precision == MV_PRECISION_FILTERED)
    return multi ? clip_kernel<T, MV_PRECISION_FILTERED, true, false>
                 : (box ? clip_kernel<T, MV_PRECISION_FILTERED, false, true>
                        : clip_kernel<T, MV_PRECISION_FILTERED, false, false>);
  return multi ? clip_kernel<T, MV_PRECISION_FP64, true, false>
               : (box ? clip_kernel<T, MV_PRECISION_FP64, false, true>
                      : clip_kernel<T, MV_PRECISION_FP64, false, false>);
}

template <class T>
static size_t clip_smem(int precision) {
  return (precision == MV_PRECISION_FILTERED ? sizeof(typename CellOf<T, MV_PRECISION_FILTERED>::type)
                                             : sizeof(typename CellOf<T, MV_PRECISION_FP64>::type)) * T::NG * T::WARPS;
}

template <class T>
static int clip_occupancy(int precision) {
  const size_t smem = clip_smem<T>(precision);
  auto k = clip_fn<T>(precision, false, false);
  int nb = 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, 32 * T::WARPS, smem) != cudaSuccess) return 0;
  return nb;
}

// Resident blocks per SM of the clip kernel (wide: the second round's tier).
int clip_blocks_per_sm(int precision, bool wide) {
  return wide ? clip_occupancy<ClipWide>(precision) : clip_occupancy<ClipFirst>(precision);
}

// Cells a block of the wide tier works on at a time.
int clip_cells_per_block() { return ClipWide::WARPS * ClipWide::NG; }

template <class T>
static cudaError_t launch_clip_t(const Job& J, StageJob SJ, const JobTable& TB, bool uneven, int resident,
                                 cudaStream_t st) {
  // four cells per warp once the resident grid is full; a smaller build leaves groups idle
  // and finishes sooner, since lockstep waits for the longest of a warp's cells (1,000 cells:
  // 0.141 ms with four per warp, 0.093 ms with one).  Lists of very uneven length (uneven: the
  // wide round of a build with dense cells) are built one per warp for longer, up to six cells
  // for each resident warp (8,100 cells of 60,000 clustered generators: all clip kernels 1.70
  // ms with four per warp, 1.59 with one; 10,900 cells: 2.01 and 2.01, 22,400: 3.39 and 3.57)
  const int64_t warps = (int64_t)resident * T::WARPS;
  SJ.per_warp = T::NG;
  while (SJ.per_warp > 1 && SJ.nitems <= warps * (SJ.per_warp / 2)) SJ.per_warp /= 2;
  if (uneven && SJ.nitems <= 6 * warps) SJ.per_warp = 1;
  const int64_t need = (SJ.nitems + SJ.per_warp - 1) / SJ.per_warp;
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(resident, (need + T::WARPS - 1) / T::WARPS));
  const size_t smem = clip_smem<T>(J.precision);
  auto k = clip_fn<T>(J.precision, TB.jobs != nullptr, SJ.box != 0);
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<blocks, 32 * T::WARPS, smem, st>>>(J, SJ, TB);
  return cudaGetLastError();
}

// The clip kernel over SJ's cells, at most `resident` blocks (wide: the second round's
// tier; uneven: lists of very different lengths).
cudaError_t launch_clip(const Job& J, const StageJob& SJ, const JobTable& TB, bool wide, bool uneven, int resident,
                        cudaStream_t st) {
  return wide ? launch_clip_t<ClipWide>(J, SJ, TB, uneven, resident, st)
              : launch_clip_t<ClipFirst>(J, SJ, TB, uneven, resident, st);
}

}  // namespace mv
