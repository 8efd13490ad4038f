// Blocked back-transform of the tridiagonal eigenvectors (compact WY form,
// LAPACK larfb order): the reflectors H_i0 ... H_i0+31 of one block are
// I - V T V^T (T from k_wy_factor), so a block costs Z <- Z - V (T (V^T Z)),
// blocks applied from the last to the first.
//
// A CTA takes MV eigenvectors of one system and keeps them in shared memory
// for the whole pass; V of the block beside them, reflector-major as it lies
// in the matrix (reflector i is row i), so that it arrives by asynchronous
// copies of contiguous elements.  All three products run as 8 x 8 x 4 FP64
// tensor tiles:
//   Y = V^T Z   one 8 x 8 tile per warp, over all rows in ascending order
//   W = T Y     one tile per warp
//   Z -= V W    8-row blocks dealt to the warps, W's fragments in registers
// Every element is summed in ascending order of its contraction index
// whatever the slice width, the chunking and the number of systems.
// Leading dimensions are 4 modulo 16 doubles: the fragment loads of every
// product are free of bank conflicts.
//
// What bounds it: with many systems the FP64 tensor pipe and the copies of V
// (two CTAs per SM run each other's copies and products side by side); with
// few, the chain of blocks (three barriers and two dependent products each),
// which is why the next block's V is then copied ahead.  Measured (B200): 361
// systems of 212 orbitals and 106 vectors 376 us (757 us with the vectors in
// global memory), one of 252 and 95 vectors 36 us (124 us with scalar FMAs),
// twelve of 900 and 450 vectors 1.5 ms (8.0 ms).
#include <algorithm>

#include "kernels.cuh"

namespace xtb {
namespace {

constexpr int WB = 32;            // reflectors per block
constexpr int kThreads = 256;
constexpr int kPT = WB + 4;       // leading dimension of T

__host__ __device__ constexpr int pad4(int n) { return (n + 11) / 16 * 16 + 4; }   // >= n, 4 modulo 16
__host__ __device__ constexpr int ldz(int n) { return pad4(n + 8); }               // rows are read in eights
template <int MV>
__host__ __device__ constexpr int ldy() { return pad4(MV); }

__device__ __forceinline__ void copy8(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Rows r0 .. r0+rows-1 of the block's V into Vt[c * ld + r - r0] (rows a
// multiple of eight; the unit diagonal, the zeros above it and past row L or
// reflector k are plain stores), one commit group.
__device__ __forceinline__ void fetch_v(const double* a, int n, int i0, int k, int L, int r0, int rows,
                                        double* Vt, int ld) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < WB; c += kThreads / 32) {
    const double* refl = a + (int64_t)(i0 + c) * n + i0 + 1;
    double* dst = Vt + c * ld - r0;
    for (int r = r0 + lane; r < r0 + rows; r += 32) {
      if (c < k && r > c && r < L) copy8(dst + r, refl + r);
      else dst[r] = (c < k && r == c) ? 1.0 : 0.0;
    }
  }
  copies_commit();
}

// One CTA's buffers and its thread's place in the tiles.
template <int MV>
struct Slice {
  static constexpr int NT = MV / 8;   // vector blocks
  static_assert(4 * NT <= kThreads / 32, "one warp per tile of Y");
  static constexpr int PY = ldy<MV>();
  double *Z, *T, *Y, *W;
  int pz, lane, warp, gq, tq;
  double y[2];

  // Warp w < 4 NT owns the tile of reflectors 8 (w & 3) .. and vectors
  // 8 (w >> 2) .. of Y, and sums it over all rows in ascending order.
  __device__ __forceinline__ bool owns_y() const { return 4 * NT >= kThreads / 32 || warp < 4 * NT; }
  __device__ __forceinline__ void clear() { y[0] = y[1] = 0.0; }
  // y += V^T Z over `rows` rows whose first is row z0 of Z
  __device__ __forceinline__ void accumulate(const double* Vt, int ld, int rows, int z0) {
    if (!owns_y()) return;
    const double* v = Vt + ((warp & 3) * 8 + gq) * ld + tq;
    const double* z = Z + ((warp >> 2) * 8 + gq) * pz + z0 + tq;
    for (int r = 0; r < rows; r += 8) {
      mma_f64(y, v[r], z[r]);
      mma_f64(y, v[r + 4], z[r + 4]);
    }
  }
  // W = T Y; ends with a barrier
  __device__ __forceinline__ void apply_t() {
    if (owns_y()) {
      double* dst = Y + ((warp & 3) * 8 + gq) * PY + (warp >> 2) * 8 + 2 * tq;
      dst[0] = y[0];
      dst[1] = y[1];
    }
    __syncthreads();
    if (owns_y()) {
      const int p0 = (warp & 3) * 8, j0 = (warp >> 2) * 8;
      double w[2] = {0.0, 0.0};
      // T is upper triangular: columns from p0 on
#pragma unroll
      for (int q = 0; q < WB; q += 4)
        if (q >= p0) mma_f64(w, T[(p0 + gq) * kPT + q + tq], Y[(q + tq) * PY + j0 + gq]);
      W[(p0 + gq) * PY + j0 + 2 * tq] = w[0];
      W[(p0 + gq) * PY + j0 + 2 * tq + 1] = w[1];
    }
    __syncthreads();
  }
  // Z -= V W over `rows` rows whose first is row z0 of Z
  __device__ __forceinline__ void update(const double* Vt, int ld, int rows, int z0) {
    double aw[NT][WB / 4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int q = 0; q < WB / 4; ++q) aw[t][q] = W[(4 * q + tq) * PY + t * 8 + gq];
    for (int r = warp * 8; r < rows; r += kThreads / 32 * 8) {
      double d[NT][2];
#pragma unroll
      for (int t = 0; t < NT; ++t) d[t][0] = d[t][1] = 0.0;
#pragma unroll
      for (int q = 0; q < WB / 4; ++q) {
        const double bv = Vt[(4 * q + tq) * ld + r + gq];
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_f64(d[t], aw[t][q], bv);
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        double* z = Z + (t * 8 + gq) * pz + z0 + r + 2 * tq;
        z[0] -= d[t][0];
        z[1] -= d[t][1];
      }
    }
  }
  __device__ __forceinline__ void load_t(const double* tf, int b) {
    for (int idx = threadIdx.x; idx < WB * WB; idx += kThreads)
      T[(idx / WB) * kPT + idx % WB] = tf[(int64_t)b * WB * WB + idx];
  }
  // vectors m of n elements between global memory and Z, zeros beyond
  __device__ __forceinline__ void load_z(const double* g, int m, int n) {
    for (int v = warp; v < MV; v += kThreads / 32)
      for (int r = lane; r < pz; r += 32) Z[v * pz + r] = v < m && r < n ? g[(int64_t)v * n + r] : 0.0;
  }
  __device__ __forceinline__ void store_z(double* g, int m, int n) {
    for (int v = warp; v < m; v += kThreads / 32)
      for (int r = lane; r < n; r += 32) g[(int64_t)v * n + r] = Z[v * pz + r];
  }
};

template <int MV>
__device__ __forceinline__ Slice<MV> make_slice(double* sm, int n) {
  Slice<MV> s;
  s.pz = ldz(n);
  s.Z = sm;
  s.T = s.Z + MV * s.pz;
  s.Y = s.T + WB * kPT;
  s.W = s.Y + WB * Slice<MV>::PY;
  s.lane = threadIdx.x & 31;
  s.warp = threadIdx.x >> 5;
  s.gq = s.lane >> 2;
  s.tq = s.lane & 3;
  return s;
}
template <int MV>
constexpr size_t slice_doubles(int n) {
  return (size_t)MV * ldz(n) + WB * kPT + 2 * WB * Slice<MV>::PY;
}

// V of a whole block in shared memory; with two buffers the next block's V
// is copied while this one is applied.  Grid (slices of MV vectors, systems);
// the count of a system's vectors is set on the device, so a CTA takes every
// gridDim.x-th slice until all are done.
template <int MV>
__global__ void __launch_bounds__(kThreads, 2) k_backtransform(EigArgs g, int buffers) {
  extern __shared__ double sm[];
  const int s = g.list[blockIdx.y];
  if (g.only != nullptr && g.only[s] == 0) return;
  const int n = g.nao[s];
  const int mt = g.all_vectors ? n : g.nvec[s];
  const int nr = n - 2;
  if (nr <= 0) return;
  const double* a = g.A + g.mat_off[s];
  const double* tf = g.scratch + g.scratch_off[s] + wy_t_offset(n);
  Slice<MV> sl = make_slice<MV>(sm, n);
  const int ld = ldz(n);
  double* V = sm + slice_doubles<MV>(n);
  const int nblk = (nr + WB - 1) / WB;
  auto fetch = [&](int b, double* dst) {
    const int i0 = b * WB, L = n - i0 - 1;
    fetch_v(a, n, i0, min(WB, nr - i0), L, 0, (L + 7) / 8 * 8, dst, ld);
  };
  for (int jbeg = blockIdx.x * MV; jbeg < mt; jbeg += gridDim.x * MV) {
    const int m = min(mt - jbeg, MV);
    double* gZ = g.Z + g.mat_off[s] + (int64_t)jbeg * n;
    __syncthreads();
    fetch(nblk - 1, V);
    sl.load_z(gZ, m, n);
    for (int it = 0; it < nblk; ++it) {
      const int b = nblk - 1 - it, i0 = b * WB;
      const int rows = (n - i0 - 1 + 7) / 8 * 8;
      double* Vt = V + (buffers == 2 && (it & 1) ? WB * ld : 0);
      sl.load_t(tf, b);
      if (buffers == 2 && b > 0) {
        fetch(b - 1, V + (it & 1 ? 0 : WB * ld));
        copies_wait<1>();   // this block's copies are done, the next one's may fly
      } else {
        copies_wait<0>();
      }
      __syncthreads();
      sl.clear();
      sl.accumulate(Vt, ld, rows, i0 + 1);
      sl.apply_t();
      sl.update(Vt, ld, rows, i0 + 1);
      __syncthreads();
      if (buffers == 1 && b > 0) fetch(b - 1, V);
    }
    sl.store_z(gZ, m, n);
  }
}
template <int MV>
size_t block_bytes(int n, int buffers) { return (slice_doubles<MV>(n) + (size_t)buffers * WB * ldz(n)) * sizeof(double); }

// Large systems, whose block of V does not fit beside the vectors: V arrives
// in chunks of 64 rows, once for Y and once for Z, the next chunk copied while
// this one is used.
constexpr int kChunk = 64;
constexpr int kLdChunk = pad4(kChunk);
template <int MV>
__global__ void __launch_bounds__(kThreads) k_backtransform_rows(EigArgs g) {
  extern __shared__ double sm[];
  const int s = g.list[blockIdx.y];
  if (g.only != nullptr && g.only[s] == 0) return;
  const int n = g.nao[s];
  const int mt = g.all_vectors ? n : g.nvec[s];
  const int nr = n - 2;
  if (nr <= 0) return;
  const double* a = g.A + g.mat_off[s];
  const double* tf = g.scratch + g.scratch_off[s] + wy_t_offset(n);
  Slice<MV> sl = make_slice<MV>(sm, n);
  double* V = sm + slice_doubles<MV>(n);
  const int nblk = (nr + WB - 1) / WB;
  auto chunks = [&](int b) { return (n - b * WB - 1 + kChunk - 1) / kChunk; };
  auto rows_of = [&](int b, int ch) { return min(kChunk, (n - b * WB - 1 - ch * kChunk + 7) / 8 * 8); };
  auto fetch = [&](int b, int ch, double* dst) {
    const int i0 = b * WB;
    fetch_v(a, n, i0, min(WB, nr - i0), n - i0 - 1, ch * kChunk, rows_of(b, ch), dst, kLdChunk);
  };
  for (int jbeg = blockIdx.x * MV; jbeg < mt; jbeg += gridDim.x * MV) {
    const int m = min(mt - jbeg, MV);
    double* gZ = g.Z + g.mat_off[s] + (int64_t)jbeg * n;
    __syncthreads();
    int stage = 0;
    fetch(nblk - 1, 0, V);
    sl.load_z(gZ, m, n);
    // the chunk in `stage` is waited for and the following one copied ahead
    auto turn = [&](int nb, int nch) {
      const double* cur = V + stage * WB * kLdChunk;
      copies_wait<0>();
      __syncthreads();
      stage ^= 1;
      if (nb >= 0) fetch(nb, nch, V + stage * WB * kLdChunk);
      return cur;
    };
    for (int b = nblk - 1; b >= 0; --b) {
      const int i0 = b * WB, nch = chunks(b);
      sl.load_t(tf, b);
      sl.clear();
      for (int ch = 0; ch < nch; ++ch) {
        const double* Vt = ch + 1 < nch ? turn(b, ch + 1) : turn(b, 0);
        sl.accumulate(Vt, kLdChunk, rows_of(b, ch), i0 + 1 + ch * kChunk);
      }
      sl.apply_t();
      for (int ch = 0; ch < nch; ++ch) {
        const double* Vt = ch + 1 < nch ? turn(b, ch + 1) : turn(b - 1, 0);
        sl.update(Vt, kLdChunk, rows_of(b, ch), i0 + 1 + ch * kChunk);
      }
      __syncthreads();
    }
    sl.store_z(gZ, m, n);
  }
}
template <int MV>
size_t rows_bytes(int n) { return (slice_doubles<MV>(n) + 2 * WB * kLdChunk) * sizeof(double); }

template <int MV>
void launch_block(const EigArgs& g, int count, int n, int want, int buffers, cudaStream_t stream) {
  allow_max_dynamic_smem(k_backtransform<MV>);
  k_backtransform<MV><<<dim3((want + MV - 1) / MV, count), kThreads, block_bytes<MV>(n, buffers), stream>>>(g, buffers);
}
// Slices of eight: sixteen took 851 us instead of 729 for 600 vectors of 1200.
void launch_rows(const EigArgs& g, int count, int n, int want, cudaStream_t stream) {
  constexpr int MV = 8;
  allow_max_dynamic_smem(k_backtransform_rows<MV>);
  k_backtransform_rows<MV><<<dim3((want + MV - 1) / MV, count), kThreads, rows_bytes<MV>(n), stream>>>(g);
}

}  // namespace

// The row-chunk kernel takes every system up to here (2764 orbitals: eight
// vectors beside two chunks of reflectors).
bool backtransform_fits(int max_n) { return rows_bytes<8>(max_n) <= allow_max_dynamic_smem(k_backtransform_rows<8>); }

void launch_backtransform(const EigArgs& g, int count, int max_n, int want_m, cudaStream_t stream) {
  if (count == 0) return;
  const size_t cap = std::min(allow_max_dynamic_smem(k_backtransform<8>), allow_max_dynamic_smem(k_backtransform<16>));
  // Slices of 16 vectors when they give every SM work (each pass over V then
  // serves twice the vectors), else slices of eight on more SMs, with the next
  // block's V copied ahead where it fits.  Where a block of V no longer fits
  // beside 16 vectors (541 to 652 orbitals) slices of eight still read V once:
  // 558 orbitals, 8 systems 0.37 ms instead of 0.46 in row chunks, 648 orbitals,
  // 24 systems 1.40 instead of 1.58.
  const bool many = (int64_t)count * ((want_m + 15) / 16) >= sm_count();
  if (many && block_bytes<16>(max_n, 1) <= cap) launch_block<16>(g, count, max_n, want_m, 1, stream);
  else if (!many && block_bytes<8>(max_n, 2) <= cap) launch_block<8>(g, count, max_n, want_m, 2, stream);
  else if (block_bytes<8>(max_n, 1) <= cap) launch_block<8>(g, count, max_n, want_m, 1, stream);
  else launch_rows(g, count, max_n, want_m, stream);
}

}  // namespace xtb
