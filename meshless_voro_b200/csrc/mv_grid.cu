// mv_grid.cu -- uniform grid (neighbour search), prefix sums, face ordering and the
// cell -> face CSR.
//
// Replaces RTree::bulk_load (rtree_nn.rs:6-8) with a device counting sort of the
// generators into a row-major uniform grid (SoA positions, coalesced for the shell
// gather of the cell kernel), and the serial flatten + Voronoi::finalize
// (voronoi.rs:226, 241-263) with scans and scatters.
#include <algorithm>
#include <cstdint>

#include <cub/device/device_radix_sort.cuh>

#include "mv_internal.h"

namespace mv {

// ------------------------------------------------------------ preparation --
// Generator::new (generator.rs:13-24): zero the unused coordinates.  Also records the
// extent of the generators and flags non-finite coordinates.
__device__ __forceinline__ unsigned long long ord_key(double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_val(unsigned long long k) {
  unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

__global__ void prep_kernel(const double* __restrict__ xyz, int n, int dim, double* __restrict__ gen,
                            unsigned long long* ext_keys /* [6]: min x,y,z, -max x,y,z */,
                            int* bad) {
  __shared__ unsigned long long smin[3], smax[3];
  if (threadIdx.x < 3) {
    smin[threadIdx.x] = ~0ull;
    smax[threadIdx.x] = 0ull;
  }
  __syncthreads();
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) {
    double c[3] = {xyz[3 * (int64_t)k], xyz[3 * (int64_t)k + 1], xyz[3 * (int64_t)k + 2]};
    if (dim == 1) c[1] = 0.0, c[2] = 0.0;
    if (dim == 2) c[2] = 0.0;
    bool fin = true;
    for (int i = 0; i < 3; i++) {
      gen[3 * (int64_t)k + i] = c[i];
      fin &= isfinite(c[i]);
    }
    if (!fin) atomicExch(bad, 1);
    for (int i = 0; i < 3; i++) {
      atomicMin(&smin[i], ord_key(c[i]));
      atomicMax(&smax[i], ord_key(c[i]));
    }
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    atomicMin(&ext_keys[threadIdx.x], smin[threadIdx.x]);
    atomicMax(&ext_keys[3 + threadIdx.x], smax[threadIdx.x]);
  }
}

// Word w of the extent that keys hold (EXT_WORDS); box: its lower and upper corner.
__device__ __forceinline__ double ext_word(const unsigned long long* keys, int w, int dim, const double* a,
                                           const double* top) {
  if (w < 6) return ord_val(keys[w]);
  bool outside = false;
  for (int i = 0; i < dim; i++) outside |= ord_val(keys[i]) < a[i] || ord_val(keys[3 + i]) > top[i];
  return outside ? 1.0 : 0.0;
}

struct Corners {
  double a[3], top[3];
};

__global__ void ext_finish_kernel(const unsigned long long* ext_keys, double* ext, int dim, Corners box,
                                  int32_t* outside /* null: not wanted */) {
  const int w = threadIdx.x;
  if (w >= EXT_WORDS) return;
  const double v = ext_word(ext_keys, w, dim, box.a, box.top);
  ext[w] = v;
  if (w == 6 && outside != nullptr) *outside = v != 0.0;
}

struct GridParams {
  int G[3];
  double a[3], inv[3];
  int dim;
};

__global__ void cell_index_kernel(const double* __restrict__ gen, int n, GridParams gp,
                                  int32_t* __restrict__ cid, int32_t* __restrict__ count) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int c[3];
  for (int i = 0; i < 3; i++) {
    double f = floor((gen[3 * (int64_t)k + i] - gp.a[i]) * gp.inv[i]);
    if (!(f >= 0.0)) f = 0.0;
    if (f > gp.G[i] - 1) f = gp.G[i] - 1;
    c[i] = (int)f;
  }
  int id = c[0] + gp.G[0] * (c[1] + gp.G[1] * c[2]);
  cid[k] = id;
  atomicAdd(count + id, 1);
}

__global__ void scatter_kernel(const double* __restrict__ gen, int n, const int32_t* __restrict__ cid,
                               const int32_t* __restrict__ start, int32_t* __restrict__ fill,
                               double* __restrict__ sx, double* __restrict__ sy,
                               double* __restrict__ sz, int32_t* __restrict__ sid) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int c = cid[k];
  int pos = start[c] + atomicAdd(fill + c, 1);
  sx[pos] = gen[3 * (int64_t)k];
  sy[pos] = gen[3 * (int64_t)k + 1];
  sz[pos] = gen[3 * (int64_t)k + 2];
  sid[pos] = k;
}

// --------------------------------------------------- dense cells (2nd level) --
// A coarse cell holding more than DENSE_MIN generators is dense: its generators are
// stored sorted by the Morton key of their position inside the cell (fkey_bits(dim) bits
// per active axis).  The cells of every level of the cell's implicit octree are then
// contiguous ranges of sorted positions, found by binary search on the keys, so a
// query scans the cells of the level that matches its radius, whatever the local
// density (Gaussian clumps span many orders of magnitude inside one coarse cell).
// Sparse cells keep key 0 and their generators in input order.
constexpr int DENSE_MIN = 32;

__global__ void dense_flag_kernel(const int32_t* __restrict__ count, int64_t ncell,
                                  int32_t* __restrict__ dflag) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  dflag[c] = count[c] > DENSE_MIN;
}

// sort key of generator k: coarse cell << FKEY_BITS | Morton key inside a dense cell
__global__ void dense_key_kernel(const double* __restrict__ gen, int n, GridParams gp,
                                 const int32_t* __restrict__ cid, const int32_t* __restrict__ dflag,
                                 unsigned long long* __restrict__ key, int32_t* __restrict__ val) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c = cid[k];
  uint32_t m = 0;
  if (dflag[c]) {
    const int bits = fkey_bits(gp.dim);
    const int cc[3] = {c % gp.G[0], (c / gp.G[0]) % gp.G[1], c / (gp.G[0] * gp.G[1])};
    uint32_t q[3] = {0u, 0u, 0u};
    for (int i = 0; i < gp.dim; i++) q[i] = fine_q(gen[3 * (int64_t)k + i], gp.a[i], gp.inv[i], cc[i], bits);
    m = morton(gp.dim, q[0], q[1], q[2]);
  }
  key[k] = ((unsigned long long)c << FKEY_BITS) | m;
  val[k] = k;
}

// sorted position s <- generator val[s]; fkey = the Morton part of its sort key
__global__ void dense_gather_kernel(const double* __restrict__ gen, int n,
                                    const unsigned long long* __restrict__ key,
                                    const int32_t* __restrict__ val, double* __restrict__ sx,
                                    double* __restrict__ sy, double* __restrict__ sz,
                                    int32_t* __restrict__ sid, uint32_t* __restrict__ fkey) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int k = val[s];
  sx[s] = gen[3 * (int64_t)k];
  sy[s] = gen[3 * (int64_t)k + 1];
  sz[s] = gen[3 * (int64_t)k + 2];
  sid[s] = k;
  fkey[s] = (uint32_t)(key[s] & ((1ull << FKEY_BITS) - 1ull));
}

// ------------------------------------------------------------------- scans --
// Exclusive scans of int32 counts into offsets, out[n] = total; blockIdx.y scans several
// arrays of one length at once.  What bounds a scan here is launches (about 3 us each where
// the arrays are small), so: up to SCAN_ONE counts one block does all (1,000 cells: 4 us,
// where the three launches of reduce, scan of the sums and final took 11); up to SCAN_SUMS
// tiles two launches, every final block adding up the sums before its own (a few KB out of
// L2 each); only beyond, where that adding would grow with the square of the tiles, a third
// launch that scans the sums.
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr int SCAN_ONE = 1024 * SCAN_ITEMS;
constexpr int SCAN_SUMS = 2048;

template <int THREADS>
__device__ __forceinline__ long long block_excl_scan(long long v, long long* total) {
  __shared__ long long wsum[THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long x = v;
  for (int o = 1; o < 32; o <<= 1) {
    long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    long long s = lane < THREADS / 32 ? wsum[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < THREADS / 32) wsum[lane] = s;
  }
  __syncthreads();
  long long wpre = w > 0 ? wsum[w - 1] : 0;
  *total = wsum[THREADS / 32 - 1];
  __syncthreads();
  return wpre + x - v;
}

// What is scanned: in[k], or in[k] + add[k], which is then also kept in sum[k].
struct ScanIn {
  const int32_t* in;
  const int32_t* add;
  int32_t* sum;
  int64_t stride;  // between the arrays of blockIdx.y
};
__device__ __forceinline__ int32_t scan_load(const ScanIn& a, int64_t k) {
  int32_t v = a.in[a.stride * blockIdx.y + k];
  if (a.add != nullptr) {
    v += a.add[k];
    a.sum[k] = v;
  }
  return v;
}

__global__ void scan_reduce_kernel(ScanIn a, int64_t n, long long* __restrict__ sums) {
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  long long s = 0;
  for (int i = 0; i < SCAN_ITEMS; i++) {
    int64_t k = base + (int64_t)i * SCAN_THREADS + threadIdx.x;
    if (k < n) s += scan_load(a, k);
  }
  long long tot;
  block_excl_scan<SCAN_THREADS>(s, &tot);
  if (threadIdx.x == 0) sums[(int64_t)gridDim.x * blockIdx.y + blockIdx.x] = tot;
}

__global__ void scan_sums_kernel(long long* sums, int nb) {
  sums += (int64_t)nb * blockIdx.y;
  long long carry = 0;
  for (int base = 0; base < nb; base += SCAN_THREADS) {
    int k = base + threadIdx.x;
    long long v = k < nb ? sums[k] : 0;
    long long tot;
    long long ex = block_excl_scan<SCAN_THREADS>(v, &tot);
    if (k < nb) sums[k] = carry + ex;
    carry += tot;
  }
}

// One tile: each thread owns SCAN_ITEMS consecutive counts; `before` is added to all.
template <int THREADS, class Out>
__device__ __forceinline__ void scan_tile(const ScanIn& a, int64_t base, int64_t n, long long before,
                                          Out* __restrict__ out) {
  int32_t v[SCAN_ITEMS];
  long long s = 0;
  for (int i = 0; i < SCAN_ITEMS; i++) {
    int64_t k = base + (int64_t)threadIdx.x * SCAN_ITEMS + i;
    v[i] = k < n ? scan_load(a, k) : 0;
    s += v[i];
  }
  long long tot;
  long long ex = block_excl_scan<THREADS>(s, &tot) + before;
  for (int i = 0; i < SCAN_ITEMS; i++) {
    int64_t k = base + (int64_t)threadIdx.x * SCAN_ITEMS + i;
    if (k < n) out[k] = (Out)ex;
    if (k == n - 1) out[n] = (Out)(ex + v[i]);
    ex += v[i];
  }
}

template <class Out>
__global__ void scan_final_kernel(ScanIn a, int64_t n, const long long* __restrict__ sums, bool scanned,
                                  Out* __restrict__ out, int64_t out_stride) {
  sums += (int64_t)gridDim.x * blockIdx.y;
  long long before = 0;
  if (scanned) {
    before = sums[blockIdx.x];
  } else {
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += SCAN_THREADS) before += sums[k];
    long long mine = before;
    block_excl_scan<SCAN_THREADS>(mine, &before);
  }
  scan_tile<SCAN_THREADS>(a, (int64_t)blockIdx.x * SCAN_TILE, n, before, out + out_stride * blockIdx.y);
}

template <class Out>
__global__ void __launch_bounds__(1024) scan_one_kernel(ScanIn a, int64_t n, Out* __restrict__ out, int64_t out_stride) {
  scan_tile<1024>(a, 0, n, 0, out + out_stride * blockIdx.y);
}

// --------------------------------------------------------------- faces/CSR --

__device__ __forceinline__ int batch_find(const int32_t* __restrict__ base, int nj, int64_t v);

// Lanes that share a cell in the kernels below: a cell owns about 8 faces (3-D).
constexpr int FACE_LANES = 8;

// Staging slots -> final positions: faces grouped by left cell in cell order, inside a
// cell in clipping-plane order (flatten!, voronoi.rs:226).  Bound by memory: 69 bytes of a
// face read and written once.  Cells come out of the pipeline in grid order, so a cell's
// faces lie together on both sides but neighbouring cells only on the written side: eight
// lanes copy a cell, so that the writes of a warp are one run and the scattered side is
// read, where a sector that is used in part costs less than one written in part.  16.5 M
// faces: 1.27 ms with a thread per face in staging order, and 0.09 ms more for the counts.
// Also counts the faces linked to their right cell (voronoi.rs:248-250: internal,
// unshifted faces; in_count null: not wanted); a batch's right indices are local to
// their tessellation (pos, nj).
__global__ void reorder_faces_kernel(FaceArrays st, int n, const int64_t* __restrict__ stage_off,
                                     const int64_t* __restrict__ face_off, FaceArrays out,
                                     int32_t* __restrict__ in_count, const int32_t* __restrict__ pos, int nj) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int g = (int)(t % FACE_LANES);
  const int64_t k = t / FACE_LANES;
  if (k >= n) return;
  const int64_t f0 = face_off[k];
  const int m = (int)(face_off[k + 1] - f0);
  if (m == 0) return;
  const int64_t q0 = stage_off[k];
  const int first = pos != nullptr && in_count != nullptr ? pos[batch_find(pos, nj, k)] : 0;
  for (int i = g; i < m; i += FACE_LANES) {
    const int32_t r = st.right[q0 + i];
    const uint8_t code = st.code[q0 + i];
    const double area = st.area[q0 + i];
    out.left[f0 + i] = (int32_t)k;
    out.right[f0 + i] = r;
    out.area[f0 + i] = area;
    out.code[f0 + i] = code;
    if (in_count != nullptr && r >= 0 && code == 13) atomicAdd(in_count + first + r, 1);
  }
  const double* c = st.centroid + 3 * q0;
  const double* v = st.normal + 3 * q0;
  double* oc = out.centroid + 3 * f0;
  double* ov = out.normal + 3 * f0;
  // four loads of each in flight per lane: 3 m is 24 where a cell owns 8 faces
  for (int b = g; b < 3 * m; b += 4 * FACE_LANES) {
    double x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (b + u * FACE_LANES < 3 * m) x[u] = c[b + u * FACE_LANES], y[u] = v[b + u * FACE_LANES];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (b + u * FACE_LANES < 3 * m) oc[b + u * FACE_LANES] = x[u], ov[b + u * FACE_LANES] = y[u];
  }
}

// A cell's connections are its incoming faces (all from lower-indexed cells, so with
// smaller face indices) followed by its own faces in order.
__global__ void conn_fill_kernel(const int32_t* __restrict__ right, const uint8_t* __restrict__ code, int n,
                                 const int64_t* __restrict__ face_off, const int64_t* __restrict__ conn_off,
                                 const int32_t* __restrict__ in_count, int32_t* __restrict__ cursor,
                                 int32_t* __restrict__ conn, const int32_t* __restrict__ pos, int nj) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int g = (int)(t % FACE_LANES);
  const int64_t k = t / FACE_LANES;
  if (k >= n) return;
  const int64_t f0 = face_off[k], f1 = face_off[k + 1];
  if (f0 == f1) return;
  const int first = pos != nullptr ? pos[batch_find(pos, nj, k)] : 0;
  int32_t* own = conn + conn_off[k] + in_count[k];
  for (int64_t f = f0 + g; f < f1; f += FACE_LANES) {
    own[f - f0] = (int32_t)f;
    const int32_t r = right[f];
    if (r >= 0 && code[f] == 13) conn[conn_off[first + r] + atomicAdd(cursor + first + r, 1)] = (int32_t)f;
  }
}

// The incoming faces in ascending order, whatever order the atomics gave.  Eight lanes rank
// a cell's faces against one another (a face's place is the number of smaller ones), up to
// four a lane; a cell with more is sorted by insertion, which was every cell's way before:
// 24 us for 1,000 cells, one thread a cell, all of it the latency of dependent accesses.
__global__ void conn_sort_kernel(const int64_t* __restrict__ conn_off,
                                 const int32_t* __restrict__ in_count, int n,
                                 int32_t* __restrict__ conn) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int g = (int)(t % FACE_LANES);
  const int64_t k = t / FACE_LANES;
  const unsigned group = 0xffu << (threadIdx.x & 24);  // the lanes of this cell
  if (k >= n) return;
  int32_t* a = conn + conn_off[k];
  const int m = in_count[k];
  if (m <= 4 * FACE_LANES) {
    int32_t v[4];
    int rank[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      v[u] = g + u * FACE_LANES < m ? a[g + u * FACE_LANES] : 0x7fffffff;
      rank[u] = 0;
    }
#pragma unroll
    for (int w = 0; w < 4; w++) {
      if (w * FACE_LANES >= m) break;
      for (int j = 0; j < FACE_LANES; j++) {
        const int32_t o = __shfl_sync(group, v[w], j, FACE_LANES);
#pragma unroll
        for (int u = 0; u < 4; u++) rank[u] += o < v[u];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (g + u * FACE_LANES < m) a[rank[u]] = v[u];
  } else if (g == 0) {
    for (int i = 1; i < m; i++) {
      int32_t v = a[i];
      int j = i - 1;
      while (j >= 0 && a[j] > v) {
        a[j + 1] = a[j];
        j--;
      }
      a[j + 1] = v;
    }
  }
}

// ------------------------------------------------------------------ batches --
// A batch concatenates its tessellations: tessellation j owns the input indices and
// sorted positions [pos[j], pos[j + 1]) and the grid cells [cbase[j], cbase[j + 1])
// (its own grid plus one empty end cell, so that its cell_start slice ends with its
// own end).  The kernels below find a point's, cell's or face's tessellation by binary
// search over these bases.
__device__ __forceinline__ int batch_find(const int32_t* __restrict__ base, int nj, int64_t v) {
  int a = 0, b = nj - 1;
  while (a < b) {
    const int m = (a + b + 1) >> 1;
    if (base[m] <= v)
      a = m;
    else
      b = m - 1;
  }
  return a;
}

__global__ void batch_ext_init_kernel(unsigned long long* ext_keys, int nj) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 6 * nj) ext_keys[i] = (i % 6) < 3 ? ~0ull : 0ull;
}

// Generator::new per tessellation (its dimensionality) and each tessellation's extent;
// a warp whose points all belong to one tessellation reduces before its atomics.
__global__ void batch_prep_kernel(const double* __restrict__ xyz, int n, const int32_t* __restrict__ pos,
                                  int nj, const BatchGrid* __restrict__ bg, double* __restrict__ gen,
                                  unsigned long long* ext_keys, int* bad) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int j = -1;
  unsigned long long kmin[3] = {~0ull, ~0ull, ~0ull}, kmax[3] = {0ull, 0ull, 0ull};
  if (k < n) {
    j = batch_find(pos, nj, k);
    const int dim = bg[j].dim;
    double c[3] = {xyz[3 * (int64_t)k], xyz[3 * (int64_t)k + 1], xyz[3 * (int64_t)k + 2]};
    if (dim == 1) c[1] = 0.0, c[2] = 0.0;
    if (dim == 2) c[2] = 0.0;
    bool fin = true;
    for (int i = 0; i < 3; i++) {
      gen[3 * (int64_t)k + i] = c[i];
      fin &= isfinite(c[i]);
      kmin[i] = kmax[i] = ord_key(c[i]);
    }
    if (!fin) atomicExch(bad, 1);
  }
  const int j0 = __shfl_sync(0xffffffffu, j, 0);
  if (__all_sync(0xffffffffu, j == j0) && j0 >= 0) {
    for (int o = 16; o > 0; o >>= 1)
      for (int i = 0; i < 3; i++) {
        kmin[i] = min(kmin[i], __shfl_xor_sync(0xffffffffu, kmin[i], o));
        kmax[i] = max(kmax[i], __shfl_xor_sync(0xffffffffu, kmax[i], o));
      }
    if (lane == 0)
      for (int i = 0; i < 3; i++) {
        atomicMin(&ext_keys[6 * j0 + i], kmin[i]);
        atomicMax(&ext_keys[6 * j0 + 3 + i], kmax[i]);
      }
  } else if (j >= 0) {
    for (int i = 0; i < 3; i++) {
      atomicMin(&ext_keys[6 * j + i], kmin[i]);
      atomicMax(&ext_keys[6 * j + 3 + i], kmax[i]);
    }
  }
}

__global__ void batch_ext_finish_kernel(const unsigned long long* ext_keys, double* ext,
                                        const BatchGrid* __restrict__ bg, int nj) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = i / EXT_WORDS;
  if (j < nj) ext[i] = ext_word(ext_keys + 6 * j, i % EXT_WORDS, bg[j].dim, bg[j].a, bg[j].top);
}

// grid cell (batch-wide index) of each generator, and the cell counts
__global__ void batch_cell_index_kernel(const double* __restrict__ gen, int n,
                                        const int32_t* __restrict__ pos, int nj,
                                        const BatchGrid* __restrict__ bg, int32_t* __restrict__ cid,
                                        int32_t* __restrict__ count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const BatchGrid& g = bg[batch_find(pos, nj, k)];
  int c[3];
  for (int i = 0; i < 3; i++) {
    double f = floor((gen[3 * (int64_t)k + i] - g.a[i]) * g.inv[i]);
    if (!(f >= 0.0)) f = 0.0;
    if (f > g.G[i] - 1) f = g.G[i] - 1;
    c[i] = (int)f;
  }
  const int id = g.cbase + c[0] + g.G[0] * (c[1] + g.G[1] * c[2]);
  cid[k] = id;
  atomicAdd(count + id, 1);
}

// sort key: batch cell << FKEY_BITS | Morton key inside a dense cell
__global__ void batch_key_kernel(const double* __restrict__ gen, int n, const int32_t* __restrict__ pos,
                                 int nj, const BatchGrid* __restrict__ bg, const int32_t* __restrict__ cid,
                                 const int32_t* __restrict__ dflag, unsigned long long* __restrict__ key,
                                 int32_t* __restrict__ val) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c = cid[k];
  uint32_t m = 0;
  if (dflag[c]) {
    const BatchGrid& g = bg[batch_find(pos, nj, k)];
    const int bits = fkey_bits(g.dim);
    const int lc = c - g.cbase;
    const int cc[3] = {lc % g.G[0], (lc / g.G[0]) % g.G[1], lc / (g.G[0] * g.G[1])};
    uint32_t q[3] = {0u, 0u, 0u};
    for (int i = 0; i < g.dim; i++) q[i] = fine_q(gen[3 * (int64_t)k + i], g.a[i], g.inv[i], cc[i], bits);
    m = morton(g.dim, q[0], q[1], q[2]);
  }
  key[k] = ((unsigned long long)c << FKEY_BITS) | m;
  val[k] = k;
}

// sorted position s <- generator val[s]; sid holds the tessellation-local index
__global__ void batch_gather_kernel(const double* __restrict__ gen, int n,
                                    const unsigned long long* __restrict__ key,
                                    const int32_t* __restrict__ val, const int32_t* __restrict__ pos,
                                    int nj, double* __restrict__ sx, double* __restrict__ sy,
                                    double* __restrict__ sz, int32_t* __restrict__ sid,
                                    uint32_t* __restrict__ fkey) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int k = val[s];
  sx[s] = gen[3 * (int64_t)k];
  sy[s] = gen[3 * (int64_t)k + 1];
  sz[s] = gen[3 * (int64_t)k + 2];
  sid[s] = k - pos[batch_find(pos, nj, k)];
  fkey[s] = (uint32_t)(key[s] & ((1ull << FKEY_BITS) - 1ull));
}

// cell_start entries of tessellation j's cells (and end cell) become local positions
__global__ void batch_local_starts_kernel(int32_t* __restrict__ start, int64_t ncell,
                                          const int32_t* __restrict__ cbase, const int32_t* __restrict__ pos,
                                          int nj) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  start[c] -= pos[batch_find(cbase, nj, c)];
}

// a tessellation without dense cells takes the one-level search, as it would by itself
__global__ void batch_levels_kernel(Job* __restrict__ jobs, const int32_t* __restrict__ dprefix,
                                    const int32_t* __restrict__ cbase, int nj) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nj || dprefix[cbase[j + 1]] != dprefix[cbase[j]]) return;
  jobs[j].dprefix = nullptr;
  jobs[j].cell_dense = nullptr;
  jobs[j].fkey = nullptr;
}

// first face and first connection of each tessellation (j = nj: the totals)
__global__ void batch_bases_kernel(const int64_t* __restrict__ face_off, const int64_t* __restrict__ conn_off,
                                   const int32_t* __restrict__ pos, int nj, int64_t* __restrict__ fbase,
                                   int64_t* __restrict__ cbase_conn) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j > nj) return;
  fbase[j] = face_off[pos[j]];
  if (conn_off != nullptr) cbase_conn[j] = conn_off[pos[j]];
}

// faces: left becomes local; CSR: offsets and face indices become local
__global__ void batch_local_faces_kernel(int32_t* __restrict__ left, int64_t F,
                                         const int32_t* __restrict__ pos, int nj) {
  const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= F) return;
  left[f] -= pos[batch_find(pos, nj, left[f])];
}

__global__ void batch_local_conn_kernel(int64_t* __restrict__ conn_off,
                                        const int32_t* __restrict__ conn_count,
                                        int32_t* __restrict__ conn, int n, const int32_t* __restrict__ pos,
                                        int nj, const int64_t* __restrict__ fbase,
                                        const int64_t* __restrict__ cbase_conn) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const int j = batch_find(pos, nj, c);
  const int64_t o = conn_off[c];
  const int32_t fb = (int32_t)fbase[j];
  for (int i = 0; i < conn_count[c]; i++) conn[o + i] -= fb;
  conn_off[c] = o - cbase_conn[j];
}

// ---------------------------------------------------------------- launchers --
static inline int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

void launch_prep(const double* xyz, int n, int dim, const double anchor[3], const double width[3], double* gen,
                 unsigned long long* ext_keys, double* ext, int32_t* outside, int* bad, cudaStream_t st) {
  Corners box;
  for (int i = 0; i < 3; i++) box.a[i] = anchor[i], box.top[i] = anchor[i] + width[i];
  if (n > 0) prep_kernel<<<nblk(n, 256), 256, 0, st>>>(xyz, n, dim, gen, ext_keys, bad);
  ext_finish_kernel<<<1, 32, 0, st>>>(ext_keys, ext, dim, box, outside);
}

void launch_grid(const double* gen, int n, const int G[3], const double a[3], const double inv[3],
                 int32_t* cid, int32_t* count, int32_t* start, int32_t* fill, double* sx, double* sy,
                 double* sz, int32_t* sid, long long* scan_tmp, cudaStream_t st);

size_t scan_tmp_elems(int64_t n) { return (size_t)((n + SCAN_TILE - 1) / SCAN_TILE) + 1; }

// rows scans of n counts each; tmp holds rows * scan_tmp_elems(n).  Returns the launches.
template <class Out>
static int scan_impl(const ScanIn& a, int64_t n, int rows, Out* out, int64_t out_stride, long long* tmp,
                     cudaStream_t st) {
  if (n <= 0) {
    for (int r = 0; r < rows; r++) cudaMemsetAsync(out + r * out_stride, 0, sizeof(Out), st);
    return 0;
  }
  if (n <= SCAN_ONE) {
    scan_one_kernel<Out><<<dim3(1, rows), 1024, 0, st>>>(a, n, out, out_stride);
    return 1;
  }
  const int nb = (int)((n + SCAN_TILE - 1) / SCAN_TILE);
  const bool scanned = nb > SCAN_SUMS;
  ScanIn final = a;
  if (a.add) final.in = a.sum, final.add = nullptr;  // the sums are there by then
  scan_reduce_kernel<<<dim3(nb, rows), SCAN_THREADS, 0, st>>>(a, n, tmp);
  if (scanned) scan_sums_kernel<<<dim3(1, rows), SCAN_THREADS, 0, st>>>(tmp, nb);
  scan_final_kernel<Out><<<dim3(nb, rows), SCAN_THREADS, 0, st>>>(final, n, tmp, scanned, out, out_stride);
  return 2 + scanned;
}

int scan_i32_to_i32(const int32_t* in, int64_t n, int32_t* out, long long* tmp, cudaStream_t st) {
  return scan_impl<int32_t>({in, nullptr, nullptr, 0}, n, 1, out, 0, tmp, st);
}
int scan_i32_to_i64(const int32_t* in, int64_t n, int64_t* out, long long* tmp, cudaStream_t st) {
  return scan_impl<int64_t>({in, nullptr, nullptr, 0}, n, 1, out, 0, tmp, st);
}
// `rows` arrays of n counts, `stride` apart, into offsets n + 1 apart
int scan_rows_i32_to_i64(const int32_t* in, int64_t n, int rows, int64_t stride, int64_t* out, long long* tmp,
                         cudaStream_t st) {
  return scan_impl<int64_t>({in, nullptr, nullptr, stride}, n, rows, out, n + 1, tmp, st);
}

void launch_grid(const double* gen, int n, const int G[3], const double a[3], const double inv[3],
                 int32_t* cid, int32_t* count, int32_t* start, int32_t* fill, double* sx, double* sy,
                 double* sz, int32_t* sid, long long* scan_tmp, cudaStream_t st) {
  GridParams gp;
  for (int i = 0; i < 3; i++) gp.G[i] = G[i], gp.a[i] = a[i], gp.inv[i] = inv[i];
  gp.dim = 3;
  int64_t ncell = (int64_t)G[0] * G[1] * G[2];
  if (n > 0) cell_index_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, gp, cid, count);
  scan_i32_to_i32(count, ncell, start, scan_tmp, st);
  if (n > 0) scatter_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, cid, start, fill, sx, sy, sz, sid);
}

// First half of the two-level grid: coarse cell index, counts, starts and the dense
// cells (flags and their running count).  The host reads the number of dense cells,
// then calls launch_grid_dense (or scatters coarse-only).  Returns the launches.
int launch_grid_coarse(const double* gen, int n, const int G[3], const double a[3],
                       const double inv[3], int32_t* cid, int32_t* count, int32_t* start,
                       int32_t* dflag, int32_t* dprefix, int dim, long long* scan_tmp, cudaStream_t st) {
  GridParams gp;
  for (int i = 0; i < 3; i++) gp.G[i] = G[i], gp.a[i] = a[i], gp.inv[i] = inv[i];
  gp.dim = dim;
  const int64_t ncell = (int64_t)G[0] * G[1] * G[2];
  if (n > 0) cell_index_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, gp, cid, count);
  int launches = 2 + scan_i32_to_i32(count, ncell, start, scan_tmp, st);
  dense_flag_kernel<<<nblk(ncell, 256), 256, 0, st>>>(count, ncell, dflag);
  return launches + scan_i32_to_i32(dflag, ncell, dprefix, scan_tmp, st);
}

// Scratch bytes of launch_grid_dense's radix sort.
size_t grid_dense_sort_bytes(int n, int64_t ncell) {
  size_t bytes = 0;
  int end_bit = FKEY_BITS;
  while ((1ll << (end_bit - FKEY_BITS)) < ncell) end_bit++;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned long long*)nullptr,
                                  (unsigned long long*)nullptr, (const int32_t*)nullptr,
                                  (int32_t*)nullptr, n, 0, end_bit);
  return bytes;
}

// Second half when some cells are dense: one stable radix sort of (cell, Morton key)
// pairs orders the generators by coarse cell and, inside dense cells, by key.
cudaError_t launch_grid_dense(const double* gen, int n, const int G[3], const double a[3],
                              const double inv[3], int dim, const int32_t* cid, const int32_t* dflag,
                              unsigned long long* key_a, unsigned long long* key_b, int32_t* val_a,
                              int32_t* val_b, void* sort_tmp, size_t sort_bytes, double* sx,
                              double* sy, double* sz, int32_t* sid, uint32_t* fkey, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  GridParams gp;
  for (int i = 0; i < 3; i++) gp.G[i] = G[i], gp.a[i] = a[i], gp.inv[i] = inv[i];
  gp.dim = dim;
  const int64_t ncell = (int64_t)G[0] * G[1] * G[2];
  int end_bit = FKEY_BITS;
  while ((1ll << (end_bit - FKEY_BITS)) < ncell) end_bit++;
  dense_key_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, gp, cid, dflag, key_a, val_a);
  cudaError_t e = cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, key_a, key_b, val_a, val_b,
                                                  n, 0, end_bit, st);
  if (e != cudaSuccess) return e;
  dense_gather_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, key_b, val_b, sx, sy, sz, sid, fkey);
  return cudaGetLastError();
}

void launch_scatter(const double* gen, int n, const int32_t* cid, const int32_t* start,
                    int32_t* fill, double* sx, double* sy, double* sz, int32_t* sid, cudaStream_t st) {
  if (n > 0) scatter_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, cid, start, fill, sx, sy, sz, sid);
}

void launch_reorder(const FaceArrays& stage, int n, const int64_t* stage_off, const int64_t* face_off,
                    const FaceArrays& out, int32_t* in_count, const int32_t* pos, int nj, cudaStream_t st) {
  if (n > 0)
    reorder_faces_kernel<<<nblk((int64_t)FACE_LANES * n, 256), 256, 0, st>>>(stage, n, stage_off, face_off, out,
                                                                             in_count, pos, nj);
}

// conn_count[k] = own + incoming faces of cell k, conn_off = their scan.  Returns the launches.
int launch_csr_offsets(const int32_t* face_count, const int32_t* in_count, int64_t n, int32_t* conn_count,
                       int64_t* conn_off, long long* scan_tmp, cudaStream_t st) {
  return scan_impl<int64_t>({face_count, in_count, conn_count, 0}, n, 1, conn_off, 0, scan_tmp, st);
}

void launch_csr_fill(const FaceArrays& f, const int64_t* face_off, const int64_t* conn_off,
                     const int32_t* in_count, int32_t* cursor, int n, int32_t* conn, const int32_t* pos, int nj,
                     cudaStream_t st) {
  if (n <= 0) return;
  const int nb = nblk((int64_t)FACE_LANES * n, 256);
  conn_fill_kernel<<<nb, 256, 0, st>>>(f.right, f.code, n, face_off, conn_off, in_count, cursor, conn, pos, nj);
  conn_sort_kernel<<<nb, 256, 0, st>>>(conn_off, in_count, n, conn);
}

// ------------------------------------------------------------ batch launchers --
// Returns the launches.
int launch_batch_grid(const double* xyz, int n, const int32_t* pos, const int32_t* cbase, int nj,
                      const BatchGrid* bg, int64_t ncell, double* gen, unsigned long long* ext_keys,
                      double* ext, int* bad, int32_t* cid, int32_t* count, int32_t* start,
                      int32_t* dflag, int32_t* dprefix, long long* scan_tmp, cudaStream_t st) {
  batch_ext_init_kernel<<<nblk(6 * (int64_t)nj, 256), 256, 0, st>>>(ext_keys, nj);
  if (n > 0) batch_prep_kernel<<<nblk(n, 256), 256, 0, st>>>(xyz, n, pos, nj, bg, gen, ext_keys, bad);
  batch_ext_finish_kernel<<<nblk(EXT_WORDS * (int64_t)nj, 256), 256, 0, st>>>(ext_keys, ext, bg, nj);
  if (n > 0) batch_cell_index_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, pos, nj, bg, cid, count);
  const int launches = 5 + scan_i32_to_i32(count, ncell, start, scan_tmp, st);
  dense_flag_kernel<<<nblk(ncell, 256), 256, 0, st>>>(count, ncell, dflag);
  return launches + scan_i32_to_i32(dflag, ncell, dprefix, scan_tmp, st);
}

size_t batch_sort_bytes(int n, int64_t ncell) { return grid_dense_sort_bytes(n, ncell); }

cudaError_t launch_batch_sort(const double* gen, int n, const int32_t* pos, const int32_t* cbase, int nj,
                              const BatchGrid* bg, int64_t ncell, const int32_t* cid, const int32_t* dflag,
                              unsigned long long* key_a, unsigned long long* key_b, int32_t* val_a,
                              int32_t* val_b, void* sort_tmp, size_t sort_bytes, double* sx, double* sy,
                              double* sz, int32_t* sid, uint32_t* fkey, int32_t* start, cudaStream_t st) {
  if (n > 0) {
    int end_bit = FKEY_BITS;
    while ((1ll << (end_bit - FKEY_BITS)) < ncell) end_bit++;
    batch_key_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, pos, nj, bg, cid, dflag, key_a, val_a);
    cudaError_t e = cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, key_a, key_b, val_a, val_b, n, 0,
                                                    end_bit, st);
    if (e != cudaSuccess) return e;
    batch_gather_kernel<<<nblk(n, 256), 256, 0, st>>>(gen, n, key_b, val_b, pos, nj, sx, sy, sz, sid, fkey);
  }
  batch_local_starts_kernel<<<nblk(ncell, 256), 256, 0, st>>>(start, ncell, cbase, pos, nj);
  return cudaGetLastError();
}

void launch_batch_levels(Job* jobs, const int32_t* dprefix, const int32_t* cbase, int nj, cudaStream_t st) {
  batch_levels_kernel<<<nblk(nj, 256), 256, 0, st>>>(jobs, dprefix, cbase, nj);
}

void launch_batch_localize(FaceArrays& f, int64_t F, const int64_t* face_off, int64_t* conn_off,
                           const int32_t* conn_count, int32_t* conn, int n, const int32_t* pos, int nj,
                           int64_t* fbase, int64_t* cbase_conn, cudaStream_t st) {
  batch_bases_kernel<<<nblk(nj + 1, 256), 256, 0, st>>>(face_off, conn_off, pos, nj, fbase, cbase_conn);
  if (F > 0) batch_local_faces_kernel<<<nblk(F, 256), 256, 0, st>>>(f.left, F, pos, nj);
  if (conn_off != nullptr && n > 0)
    batch_local_conn_kernel<<<nblk(n, 256), 256, 0, st>>>(conn_off, conn_count, conn, n, pos, nj, fbase,
                                                          cbase_conn);
}

}  // namespace mv
