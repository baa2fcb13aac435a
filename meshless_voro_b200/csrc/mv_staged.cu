// mv_staged.cu -- the staged cell pipeline: shell and integral kernels.
//
// The same per-cell construction as the fused kernel (mv_cells.cu), split in three
// kernels over a chunk of cells so that each kernel keeps a small instruction
// footprint and its own occupancy:
//   1. shell_kernel gathers each cell's first neighbour shell (rtree_nn.rs:10-240
//      up to the initial radius) and writes it sorted to a candidate list;
//   2. clip_kernel (mv_clip.cu) runs ConvexCell::build (convex_cell.rs:316-356) over the
//      list and writes the finished cell (planes, vertices in the reference's order) to a
//      record;
//   3. integrate_kernel evaluates the integrals and emits the faces
//      (voronoi_cell.rs:40-100) from the record.
// A cell whose list does not decide it (the stream continues past the first shell,
// or the shell overflowed) goes to a retry list that the fused kernel builds from
// scratch afterwards, so every cell still sees the reference's full neighbour stream.
#include <cfloat>
#include <cstdint>

#include "mv_cell_common.cuh"

namespace mv {

constexpr int SHELL_CMAX = 128;
constexpr int SHELL_MIN = 64;  // first shells below this many candidates are widened
constexpr int SHELL_WARPS = 4;
#ifndef MV_SHELL_MINB
#define MV_SHELL_MINB 8
#endif
constexpr int INT_WARPS = 4;
#ifndef MV_INT_STEP
#define MV_INT_STEP 10
#endif
constexpr int INT_STEP = MV_INT_STEP;  // vertices per step of the integral kernel
#ifndef MV_INT_MINB
#define MV_INT_MINB 7
#endif
using TierClip = Tier<64, 64, SHELL_CMAX, 8, uint8_t, 1>;  // capacity of a record

// sorted position of processing item `item` of a chunk
__device__ __forceinline__ int stage_pos(const StageJob& SJ, int item) {
  return SJ.order != nullptr ? __ldg(SJ.order + SJ.item0 + item) : SJ.item0 + item;
}

// ------------------------------------------------------------------- shell --
// Bitonic sort of 32 * EPL distinct 32-bit keys in registers (element i = lane + 32 e in
// slot e of every lane): one shuffle and one minimum or maximum per exchange.
template <int EPL>
__device__ __forceinline__ void sort_regs_key(uint32_t (&key)[EPL], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * EPL; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int e = 0; e < EPL; e++) {
          const int pe = e ^ (j >> 5);
          if (pe > e) {
            const bool asc = ((32 * e) & k) == 0;
            const uint32_t a = key[e], b = key[pe];
            key[e] = asc ? min(a, b) : max(a, b);
            key[pe] = asc ? max(a, b) : min(a, b);
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < EPL; e++) {
          const uint32_t o = __shfl_xor_sync(FULL, key[e], j);
          const bool low = ((((lane + 32 * e) & k) == 0) == ((lane & j) == 0));
          key[e] = low ? min(key[e], o) : max(key[e], o);
        }
      }
    }
  }
}

// Sorts the gathered shell (cnt <= 32 EPL entries with squared distances below R2; B.tie
// holds the shift codes) in registers and writes it as sorted position * 27 + shift code;
// returns whether the nearest entry is the generator itself (sorted position spos, no
// shift).  An entry's key is its squared distance as a 25-bit fraction of R2 above its
// index in the shell: one word to compare and move per entry (a distance word and a list
// word before; with one row pass per query, see gather_shell: 128^3 Poisson cells 10.8 ->
// 7.6 ms), which orders the entries as
// their squared distances do (the fraction is a monotone function of them) unless two
// fractions are equal (distances within 2^-25 R2, or equal as in lattice-like inputs; one
// uniform cell in some thousands); the shell is then sorted again by (squared distance,
// original index, shift code), the stream's full order.
template <int EPL>
__device__ __forceinline__ bool sort_and_write(const Job& J, const ShellBuf<SHELL_CMAX>& B, int lane,
                                               int cnt, double R2, int self, int spos, uint32_t* out) {
  uint32_t key[EPL];
  const double scale = (double)(1 << 25) / R2;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    const int i = lane + 32 * e;
    // 0 <= d2 < R2; the rounded product may reach 2^25
    const uint32_t f =
        i < cnt ? min(__double2uint_rz(__longlong_as_double((long long)B.key[i]) * scale), (1u << 25) - 1u)
                : (1u << 25) - 1u;
    key[e] = (f << 7) | (uint32_t)i;
  }
  sort_regs_key<EPL>(key, lane);
  // equal fractions end next to each other: element i against i + 1 (padding, with the
  // largest fraction and indices from cnt on, sorts behind every entry)
  bool dup = false;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    const uint32_t nx = __shfl_down_sync(FULL, key[e], 1);
    const uint32_t wrap = __shfl_sync(FULL, key[e + 1 < EPL ? e + 1 : e], 0);
    const uint32_t next = lane < 31 ? nx : wrap;
    const int i = lane + 32 * e;
    dup |= (i + 1 < cnt) && (key[e] >> 7) == (next >> 7);
  }
  if (__any_sync(FULL, dup)) {
    unsigned long long dkey[EPL];
    uint32_t tie[EPL];
    int32_t pos[EPL];
#pragma unroll
    for (int e = 0; e < EPL; e++) {
      const int i = lane + 32 * e;
      dkey[e] = i < cnt ? B.key[i] : ~0ull;
      tie[e] = i < cnt ? (uint32_t)__ldg(J.sid + B.cpos[i]) * 27u + B.tie[i] : ~0u;
      pos[e] = i < cnt ? B.cpos[i] : 0;
    }
    sort_regs<EPL>(dkey, tie, pos, lane);
#pragma unroll
    for (int e = 0; e < EPL; e++) {
      const int i = lane + 32 * e;
      if (i < cnt) out[i] = (uint32_t)pos[e] * 27u + tie[e] % 27u;
    }
    return (int)(__shfl_sync(FULL, tie[0], 0) / 27u) == self;
  }
  uint32_t first = 0u;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    const int i = lane + 32 * e, at = (int)(key[e] & 127u);
    const uint32_t v = (uint32_t)B.cpos[at] * 27u + B.tie[at];
    if (i < cnt) out[i] = v;
    if (e == 0) first = v;
  }
  return __shfl_sync(FULL, first, 0) == (uint32_t)spos * 27u + 13u;
}

template <int WARPS, bool MULTI, bool OUT>
__global__ void __launch_bounds__(32 * WARPS, MV_SHELL_MINB)
    shell_kernel(const __grid_constant__ Job J0, const __grid_constant__ StageJob SJ,
                 const __grid_constant__ JobTable TB) {
  __shared__ ShellBuf<SHELL_CMAX> bufs[WARPS];
  __shared__ double ext_s[EXT_WORDS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ShellBuf<SHELL_CMAX>& B = bufs[warp];
  if (threadIdx.x < EXT_WORDS) ext_s[threadIdx.x] = J0.ext[threadIdx.x];
  __syncthreads();
  for (;;) {
    int item = 0;
    if (lane == 0) item = (int)atomicAdd(SJ.work + 0, 1u);
    item = __shfl_sync(FULL, item, 0);
    if (item >= SJ.nitems) break;
    const int gpos = stage_pos(SJ, item);
    // the cell's tessellation (batch builds): its Job and its local position
    const int jb = MULTI ? job_of(TB, gpos) : 0;
    const Job& J = MULTI ? TB.jobs[jb] : J0;
    const int spos = MULTI ? gpos - __ldg(TB.pos_base + jb) : gpos;
    const double* ext = MULTI ? J.ext : ext_s;
    const int self = __ldg(J.sid + spos);
    if (J.mask != nullptr && J.mask[self] == 0) {
      if (lane == 0) SJ.info[item] = 0;
      continue;
    }
    const D3 x = load_gen(J, self);
    bool all = false;
    double R = first_radius(J, x, lane);
    int cnt = gather_shell<SHELL_CMAX, OUT, false, true>(J, B, lane, x, R, 0.0, ext, &all, 32 * SHELL_CMAX);
    // the density estimate behind R is rough where the density varies: a shell that
    // overflows the list is pulled in, one far below a uniform region's ~92 candidates
    // (too small to close most cells) is widened, a few times at most
    for (int it = 0; it < 6; it++) {
      double f;
      if (cnt > SHELL_CMAX)
        f = fmin(fmax(cbrt(0.6 * SHELL_CMAX / (double)cnt), 0.1), 0.9);
      else if (cnt < SHELL_MIN && !all)
        f = fmin(cbrt(96.0 / (double)max(cnt, 1)), 2.0);
      else
        break;
      R *= f;
      cnt = gather_shell<SHELL_CMAX, OUT, false, true>(J, B, lane, x, R, 0.0, ext, &all, 32 * SHELL_CMAX);
    }
    if (cnt > SHELL_CMAX || cnt == 0) {
      if (lane == 0) SJ.info[item] = -1;
      continue;
    }
    uint32_t* out = SJ.cand + (int64_t)item * SJ.cstride;
    bool self_first;
    if (cnt <= 32)
      self_first = sort_and_write<1>(J, B, lane, cnt, R * R, self, spos, out);
    else if (cnt <= 64)
      self_first = sort_and_write<2>(J, B, lane, cnt, R * R, self, spos, out);
    else
      self_first = sort_and_write<4>(J, B, lane, cnt, R * R, self, spos, out);
    // the first neighbour must be the generator itself (convex_cell.rs:325-329); the
    // fused kernel reports the error otherwise
    if (lane == 0) {
      SJ.info[item] = self_first ? (cnt | (all ? (1 << 30) : 0)) : -1;
      SJ.rad[item] = R;
    }
    __syncwarp();
  }
}

// The wide round: cells the first round could not close get a shell of up to WIDE_CMAX
// candidates (about eight times the first one), sorted in shared memory.  Cells the
// wide round cannot close either go to the fused kernel.
// Its radius is found by count.  In a periodic build without dense cells a cell that the
// first shell did not close has a shallow void beside it: 1.4 radii, about 250 candidates,
// close all but the few whose cell outgrows the tier, and sort in a quarter of the time
// (16,736 cells of 128^3 Poisson generators: 1.07 -> 0.40 ms, 54 cells of 4,096: 0.10 ->
// 0.06 ms).  At a wall half of a shell is empty (6,000 generators in a box: two cells stay
// open with it, and cost 0.17 ms in the fused kernel), and beside clumps a cell may need
// thousands: there a shell of two radii, about 740 candidates, closes more than it costs
// (8.4 M clustered generators: 843 ms, with the small shells 853).
constexpr int WIDE_CMAX = 1024;
constexpr int WIDE_WARPS = 4;
constexpr size_t WIDE_SMEM = sizeof(ShellBuf<WIDE_CMAX>) * WIDE_WARPS;

// Sorts the wide shell [0, n) by the squared distance rounded down to f32 (as
// sort_and_write) in place of B.key: each key becomes that 32-bit key above the
// entry's index, so one 64-bit word is compared and moved per entry.  Returns false
// when two keys are equal (the order then needs the full (key, tie) sort, over the
// original keys, which this overwrote).
template <int CMAX>
__device__ __noinline__ bool sort_shell_key32(ShellBuf<CMAX>& B, int lane, int n) {
  int np2 = 32;
  while (np2 < n) np2 <<= 1;
  for (int i = lane; i < np2; i += 32) {
    unsigned long long w = ~0ull;
    if (i < n) {
      const float k = __double2float_rd(__longlong_as_double((long long)B.key[i]));
      w = ((unsigned long long)__float_as_uint(k) << 32) | (unsigned)i;
    }
    B.key[i] = w;
  }
  __syncwarp();
  for (int k = 2; k <= np2; k <<= 1) {
    for (int jl = __ffs(k) - 2; jl >= 0; jl--) {
      const int j = 1 << jl;
      for (int i = lane; i < (np2 >> 1); i += 32) {
        const int lo = ((i >> jl) << (jl + 1)) | (i & (j - 1));
        const int hi = lo + j;
        const unsigned long long ka = B.key[lo], kb = B.key[hi];
        if ((ka > kb) == ((lo & k) == 0)) B.key[lo] = kb, B.key[hi] = ka;
      }
      __syncwarp();
    }
  }
  bool dup = false;
  for (int i = lane; i + 1 < n; i += 32) dup |= (B.key[i] >> 32) == (B.key[i + 1] >> 32);
  return !__any_sync(FULL, dup);
}

template <int WARPS, bool MULTI, bool OUT>
__global__ void __launch_bounds__(32 * WARPS, 3)
    shell_wide_kernel(const __grid_constant__ Job J0, const __grid_constant__ StageJob SJ,
                      const __grid_constant__ JobTable TB) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double ext_s[EXT_WORDS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ShellBuf<WIDE_CMAX>& B = reinterpret_cast<ShellBuf<WIDE_CMAX>*>(smem_raw)[warp];
  if (threadIdx.x < EXT_WORDS) ext_s[threadIdx.x] = J0.ext[threadIdx.x];
  __syncthreads();
  for (;;) {
    int item = 0;
    if (lane == 0) item = (int)atomicAdd(SJ.work + 0, 1u);
    item = __shfl_sync(FULL, item, 0);
    if (item >= SJ.nitems) break;
    const int gpos = stage_pos(SJ, item);
    // the cell's tessellation (batch builds): its Job and its local position
    const int jb = MULTI ? job_of(TB, gpos) : 0;
    const Job& J = MULTI ? TB.jobs[jb] : J0;
    const int spos = MULTI ? gpos - __ldg(TB.pos_base + jb) : gpos;
    const double* ext = MULTI ? J.ext : ext_s;
    const int self = __ldg(J.sid + spos);
    if (J.mask != nullptr && J.mask[self] == 0) {
      if (lane == 0) SJ.info[item] = 0;
      continue;
    }
    const D3 x = load_gen(J, self);
    bool all = false;
    const bool even = J.fkey == nullptr && J.periodic;
    const int least = even ? 128 : 384;  // widened below this many candidates
    const double aim = even ? 256.0 : 768.0;
    double R = (even ? 1.4 : 2.0) * first_radius(J, x, lane);
    int cnt = gather_shell<WIDE_CMAX, OUT>(J, B, lane, x, R, 0.0, ext, &all, 4 * WIDE_CMAX);
    for (int it = 0; it < 6; it++) {
      double f;
      if (cnt > WIDE_CMAX)
        f = fmin(fmax(cbrt(0.6 * WIDE_CMAX / (double)cnt), 0.1), 0.9);
      else if (cnt < least && !all)
        f = fmin(cbrt(aim / (double)max(cnt, 1)), 2.0);
      else
        break;
      R *= f;
      cnt = gather_shell<WIDE_CMAX, OUT>(J, B, lane, x, R, 0.0, ext, &all, 4 * WIDE_CMAX);
    }
    if (cnt > WIDE_CMAX || cnt == 0) {
      if (lane == 0) SJ.info[item] = -1;
      continue;
    }
    uint32_t* out = SJ.cand + (int64_t)item * SJ.cstride;
    uint32_t first;  // the nearest entry's tie (original index * 27 + shift code)
    if (sort_shell_key32<WIDE_CMAX>(B, lane, cnt)) {
      for (int i = lane; i < cnt; i += 32) {
        const int e = (int)(uint32_t)B.key[i];
        out[i] = (uint32_t)B.cpos[e] * 27u + B.tie[e] % 27u;
      }
      first = B.tie[(uint32_t)B.key[0]];
    } else {
      // equal keys: the same shell again (the gather is deterministic), fully sorted
      cnt = gather_shell<WIDE_CMAX, OUT>(J, B, lane, x, R, 0.0, ext, &all, 4 * WIDE_CMAX);
      sort_shell<WIDE_CMAX>(B, lane, cnt);
      for (int i = lane; i < cnt; i += 32) out[i] = (uint32_t)B.cpos[i] * 27u + B.tie[i] % 27u;
      first = B.tie[0];
    }
    if (lane == 0) {
      const bool self_first = (int)(first / 27u) == self;
      SJ.info[item] = self_first ? (cnt | (all ? (1 << 30) : 0)) : -1;
      SJ.rad[item] = R;
    }
    __syncwarp();
  }
}

// --------------------------------------------------------------- integrals --
template <class T, int WARPS, bool MULTI>
__global__ void __launch_bounds__(32 * WARPS, MV_INT_MINB)
    integrate_kernel(const __grid_constant__ Job J0, const __grid_constant__ StageJob SJ,
                     const __grid_constant__ JobTable TB) {
  __shared__ TetScratch<INT_STEP, T::PMAX> scratch[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = lane; i < T::PMAX; i += 32) scratch[warp].pm[i] = 0u;
  __syncwarp();
  unsigned done = 0;
  for (;;) {
    int item = 0;
    if (lane == 0) item = (int)atomicAdd(SJ.work + 2, 1u);
    item = __shfl_sync(FULL, item, 0);
    if (item >= SJ.nitems) break;
    const int64_t off = SJ.rec_off[item];
    if (off < 0) continue;
    const int gpos = stage_pos(SJ, item);
    const int jb = MULTI ? job_of(TB, gpos) : 0;
    const Job& J = MULTI ? TB.jobs[jb] : J0;
    const int spos = MULTI ? gpos - __ldg(TB.pos_base + jb) : gpos;
    const int self = __ldg(J.sid + spos);
    const D3 x = load_gen(J, self);
    const RecordView V(SJ.rec + off);
    int err = 0;
    const int res = integrate_view<T, INT_STEP>(J, V, scratch[warp], lane, self, x, V.nv, V.np, V.sr, &err);
    if (res == CELL_DONE) {
      done++;
    } else if (lane == 0) {
      if (res == CELL_FACE_OVERFLOW) {
        atomicExch(J.status + STATUS_FACE_OVERFLOW, 1);
      } else {
        atomicCAS(J.status + STATUS_CODE, 0, err);
        atomicMin(J.status + STATUS_CELL, self + J.id_base);
      }
    }
    __syncwarp();
  }
  if (lane == 0 && done) atomicAdd(J0.stats + ST_CELLS, (unsigned long long)done);
}

// ---------------------------------------------------------------- launchers --
template <class K>
static int occupancy(K k, int threads, size_t smem) {
  int nb = 0;
  if (smem > 0 &&
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, threads, smem) != cudaSuccess) return 0;
  return nb;
}

int stage_blocks_per_sm(int kernel) {
  if (kernel == 0) return occupancy(shell_kernel<SHELL_WARPS, false, false>, 32 * SHELL_WARPS, 0);
  if (kernel == 3) return occupancy(shell_wide_kernel<WIDE_WARPS, false, false>, 32 * WIDE_WARPS, WIDE_SMEM);
  return occupancy(integrate_kernel<TierClip, INT_WARPS, false>, 32 * INT_WARPS, 0);
}

__global__ void append_range_kernel(int32_t* dst, int32_t first, int32_t count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) dst[i] = first + i;
}

// dst[i] = first + i for i < count (processing positions handed to the fused kernel)
cudaError_t launch_append_range(int32_t* dst, int32_t first, int32_t count, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  append_range_kernel<<<(count + 255) / 256, 256, 0, st>>>(dst, first, count);
  return cudaGetLastError();
}

int stage_list_stride() { return SHELL_CMAX; }
int stage_wide_stride() { return WIDE_CMAX; }

int64_t stage_record_words(int np, int nv) { return rec_words(np, nv); }

template <bool MULTI, bool OUT>
static cudaError_t launch_stage_t(int kernel, const Job& J, const StageJob& SJ, const JobTable& TB,
                                  int blocks, cudaStream_t st) {
  if (kernel == 0) {
    shell_kernel<SHELL_WARPS, MULTI, OUT><<<blocks, 32 * SHELL_WARPS, 0, st>>>(J, SJ, TB);
  } else if (kernel == 3) {
    auto k = shell_wide_kernel<WIDE_WARPS, MULTI, OUT>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WIDE_SMEM);
    if (e != cudaSuccess) return e;
    k<<<blocks, 32 * WIDE_WARPS, WIDE_SMEM, st>>>(J, SJ, TB);
  } else {
    integrate_kernel<TierClip, INT_WARPS, MULTI><<<blocks, 32 * INT_WARPS, 0, st>>>(J, SJ, TB);
  }
  return cudaGetLastError();
}

// Launches stage kernel `kernel` (0 shell, 2 integrals, 3 wide shell; the clip kernel is
// launch_clip's); with a job table (TB.jobs != nullptr) over the cells of a batch.
cudaError_t launch_stage(int kernel, const Job& J, const StageJob& SJ, const JobTable& TB, int blocks,
                         cudaStream_t st) {
  if (blocks < 1) blocks = 1;
  if (TB.jobs != nullptr) return launch_stage_t<true, true>(kernel, J, SJ, TB, blocks, st);
  return J.outside ? launch_stage_t<false, true>(kernel, J, SJ, TB, blocks, st)
                   : launch_stage_t<false, false>(kernel, J, SJ, TB, blocks, st);
}

}  // namespace mv
