// Householder tridiagonalisation of systems that neither shared memory nor a
// cluster's registers hold: one thread-block cluster per system, the matrix
// in global memory (L2 resident: a 1200-orbital triangle is 5.8 MB), two
// cluster barriers per column.
//
// The trailing block's upper triangle is kept in place in the square matrix
// (row r, columns c >= r), so a column of the reduction is a contiguous row.
// Column step o, every CTA of the cluster:
//   (1) redundantly in every CTA: w_{o-1} = tau p - (tau^2/2)(p.v) v from
//       p = A^(o-1) v_{o-1}, row o of A^(o), its norm and reflector o;
//   (2) the rows o+1.. are updated with (v_{o-1}, w_{o-1}) and multiplied by
//       v_o in the same pass, in units of 8 rows x 64 columns: the units, row
//       block by row block, are cut into equal contiguous runs, one per warp
//       of the cluster, so that a row block's sums stay in registers along a
//       run and one butterfly per row block (not one per unit) adds them over
//       the lanes;
//   (3) the CTA's warps' partial products are added and each row's sum stored
//       into the CTA that adds that row's parts -- cluster barrier --, which
//       stores the total into every CTA  -- cluster barrier --.  Nothing waits
//       for a remote load.
// Outputs as the other tridiagonalisations: d, e, tau, and reflector o in row
// o of the matrix (columns o+2..n-1, v[o+1] = 1 implicit).  Row o is read by
// every CTA during step o, so its reflector is written during step o+1.
//
// What bounds it: a column costs about 3.5 us of barriers and dependent sums
// (n = 258) and, above about 500 orbitals, the units of (2): their dependent
// multiply-adds and L2 loads, which the two warps a scheduler do not hide (8
// systems of 600 to 1200 orbitals: issue active 32 % of cycles, FP64 pipe 12 %,
// L2 12 %; per issued instruction 1.4 waits for a fixed latency, 1.1 for L2, 0.8
// at barriers).  Measured (B200, one system): n = 360 1.41 ms, 600 2.90 ms, 900
// 5.8 ms, 1200 9.7 ms, 2100 33 ms; with four warps a CTA, where eight have no
// room, 2214 100 ms; the single-CTA prefix (k_tridiag_prefix + k_tridiag_smem)
// took 4.1, 17.4 and, at 1200, 126 ms.  A butterfly per unit instead of per row
// block: 38 ms instead of 13 ms at n = 1200 with eight CTAs.  Eight warps a CTA,
// two CTAs an SM: sixteen warps take the same time alone and leave no room for
// a second system (30 systems of 258: 1.19 ms instead of 2.4 ms).  128 registers
// a thread for that, with 8 bytes of spill stores.
//
// Reference behaviour: the reduction LAPACK's dsytrd performs inside dsyevd
// (model/gfn2/eigensolver.cpp:1221-1254 of the reference).
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "kernels.cuh"

namespace xtb {
namespace cg = cooperative_groups;

namespace {

constexpr int kUnitRows = 8;
constexpr int kUnitCols = 64;

// Elements of the unit whose first row starts at `row` (lane columns c and
// c + 32; cok: the column exists; rows: bit i set where row i is live).
__device__ __forceinline__ void load_unit(const double* row, int n, unsigned rows, const bool (&cok)[2],
                                          double (&a)[kUnitRows][2]) {
#pragma unroll
  for (int i = 0; i < kUnitRows; ++i) {
    const bool rok = (rows >> i) & 1u;
#pragma unroll
    for (int h = 0; h < 2; ++h) a[i][h] = rok && cok[h] ? __ldcg(row + 32 * h) : 0.0;
    row += n;
  }
}

// Updates one unit with (v, w) and multiplies it by x: the rows' sums go to
// pw, the transposed part (times xr, the rows' x; zeros where the unit lies in
// a diagonal block, which holds both triangles) to col.  A dead row or column
// has a zero element or zero x and is not stored.  The row sums are reduced by
// a butterfly reduce-scatter that leaves row (lane & 7) in every lane
// congruent to it.
__device__ __forceinline__ void apply_unit(double* row, int n, unsigned rows, const bool (&cok)[2],
                                           const double2* vwr, const double* xr, const double2 (&vwc)[2],
                                           const double (&xc)[2], double (&a)[kUnitRows][2],
                                           double (&sum)[kUnitRows], double (&col)[2]) {
#pragma unroll
  for (int i = 0; i < kUnitRows; ++i) {
    const double2 t = vwr[i];
    const double x = xr[i];
    const bool rok = (rows >> i) & 1u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double u = fma(-t.x, vwc[h].y, a[i][h]);
      u = fma(-t.y, vwc[h].x, u);
      if (rok && cok[h]) __stcg(row + 32 * h, u);
      sum[i] = fma(u, xc[h], sum[i]);
      col[h] = fma(u, x, col[h]);
    }
    row += n;
  }
}

// Sums of the rows of a unit over the lanes: a butterfly reduce-scatter that
// leaves row (lane & 7) in every lane congruent to it.
__device__ __forceinline__ double reduce_rows(double (&sum)[kUnitRows], int lane) {
#pragma unroll
  for (int sh = kUnitRows / 2; sh >= 1; sh >>= 1) {
    const bool up = (lane & sh) != 0;
#pragma unroll
    for (int k = 0; k < sh; ++k) {
      const double send = up ? sum[k] : sum[k + sh];
      const double keep = up ? sum[k + sh] : sum[k];
      sum[k] = keep + __shfl_xor_sync(0xffffffffu, send, sh);
    }
  }
#pragma unroll
  for (int x = kUnitRows; x < 32; x <<= 1) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], x);
  return sum[0];
}

__host__ __device__ constexpr int padded(int n) { return (n + kUnitRows - 1) / kUnitRows * kUnitRows; }

// Rows of an n-row vector that one CTA adds: its share of the 32-row blocks.
template <int G>
__host__ __device__ constexpr int slice_rows(int n) {
  return ((n + 31) / 32 + G - 1) / G * 32;
}

template <int G, int NW>
__global__ void __launch_bounds__(32 * NW, 2) k_tridiag_large(EigArgs g, const int32_t* list) {
  extern __shared__ double sm[];
  constexpr int NT = 32 * NW;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int s = list[blockIdx.x / G];
  // uniform over the cluster: all of its CTAs return before any barrier
  if (g.only != nullptr && g.only[s] == 0) return;
  const int n = g.nao[s];
  if (n < 3) return;   // the caller sends larger systems only
  double* A = g.A + g.mat_off[s];
  double* d = g.d + g.ao_off[s];
  double* e = g.e + g.ao_off[s];
  double* tau = g.tau + g.ao_off[s];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // vectors indexed by the global row, padded to whole units with zeros
  const int np = padded(n);
  double2* vw = reinterpret_cast<double2*>(sm);   // (v, w) of the reflector being applied
  double* xn = sm + 2 * np;                       // the row being reduced: v / scale but for x[o+1]; 0 up to o
  double* p = xn + np;                            // A x', summed over the cluster
  double* recv = p + np;                           // G slices: the CTAs' parts of the rows this CTA adds
  const int slice = slice_rows<G>(n);
  double* priv = recv + G * slice;                // the warps' partial products, np each
  double* first = priv + NW * np;                 // per warp: the first row block's x; then zeros
  __shared__ double red[32];
  __shared__ double dots[G * NW];                 // the cluster's warps' parts of p.x'
  __shared__ double s_alpha;
  for (int k = tid; k < np; k += NT) {
    vw[k] = make_double2(0.0, 0.0);
    xn[k] = p[k] = 0.0;
  }
  for (int k = tid; k < NW * np + (NW + 1) * kUnitRows; k += NT) priv[k] = 0.0;
  for (int k = tid; k < G * slice; k += NT) recv[k] = 0.0;
  for (int k = tid; k < G * NW; k += NT) dots[k] = 0.0;
  double* pw = priv + warp * np;
  double* xfirst = first + warp * kUnitRows;
  const double* xzero = first + NW * kUnitRows;
  cluster.sync();

  const int J = (n + kUnitCols - 1) / kUnitCols;
  const int NB = (n + kUnitRows - 1) / kUnitRows;
  const int wg = rank * NW + warp;
  constexpr int kPer = kUnitCols / kUnitRows;
  // reflector o-1: tau and the scale that makes v = scp x with v[o] = 1
  double taup = 0.0, scp = 0.0;
  for (int o = 0; o + 1 < n; ++o) {
    const bool next = o + 2 < n;     // reflector o exists
    // This warp's run of units, row block by row block: row block rb has the
    // column blocks rb / 8 .. J - 1.  The first unit's elements do not depend
    // on this step's vectors, so they are loaded ahead of (1).
    const int lo = o + 1;
    const int rb0 = lo / kUnitRows;
    auto columns_before = [&](int k) {   // sum of i / 8 over i < k
      const int q = k / kPer, m = k % kPer;
      return kPer / 2 * q * (q - 1) + m * q;
    };
    const int skipped = columns_before(rb0);
    auto before = [&](int rb) { return J * (rb - rb0) - (columns_before(rb) - skipped); };
    int rb = rb0, u = 0, uend = 0;
    if (next) {
      const int total = before(NB);
      u = total * wg / (G * NW);
      uend = total * (wg + 1) / (G * NW);
      // the row block that holds unit u: the lanes try 32 blocks at once
      while (true) {
        const int k = rb + 1 + lane;
        const int ahead = __popc(__ballot_sync(0xffffffffu, k < NB && u >= before(k)));
        rb += ahead;
        if (ahead < 32) break;
      }
    }
    // live rows of a row block
    auto rows = [&](int rb) {
      const int r0 = rb * kUnitRows;
      unsigned m = (1u << kUnitRows) - 1u;
      if (r0 < lo) m &= m << (lo - r0);
      if (r0 + kUnitRows > n) m &= (1u << (n - r0)) - 1u;
      return m;
    };
    int jb = rb / kPer + (u - before(rb));
    unsigned live = rows(rb);
    double* row = A + (size_t)rb * kUnitRows * n + jb * kUnitCols + lane;
    bool cok[2] = {jb * kUnitCols + lane < n, jb * kUnitCols + lane + 32 < n};
    double a0[kUnitRows][2];
    if (u < uend) load_unit(row, n, live, cok, a0);
    // ---- (1) ----
    double kw = 0.0, w0 = 0.0;
    const double tp = taup * scp;      // A v = scp p, p.v = scp (p.x')
    if (o > 0) {
      double pv = 0.0;
#pragma unroll
      for (int k = 0; k < G * NW; k += 32)
        if (k + lane < G * NW) pv += dots[k + lane];
      kw = 0.5 * tp * tp * warp_sum(pv);
      w0 = fma(tp, p[o], -kw);         // v[o] = 1
    }
    double nrm = 0.0;
    for (int r = o + tid; r < n; r += NT) {
      double c = __ldcg(A + (size_t)o * n + r);
      if (o > 0) {
        const double v = r == o ? 1.0 : scp * xn[r];
        const double w = fma(tp, p[r], -kw * v);
        vw[r] = make_double2(v, w);
        c -= fma(v, w0, w);            // row o of A^(o); v[o] = 1
      }
      xn[r] = r == o ? 0.0 : c;
      if (r == o && rank == 0) d[o] = c;
      if (r == o + 1) s_alpha = c;
      if (r >= o + 2) nrm = fma(c, c, nrm);
    }
    // norm of the row: one barrier, every thread adds the warps' parts
    nrm = warp_sum(nrm);
    if (lane == 0) red[warp] = nrm;
    __syncthreads();
    nrm = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) nrm += red[w];
    const double alpha = s_alpha;
    double beta = alpha, ti = 0.0, sc = 0.0;
    if (next && nrm > 0.0) {
      beta = -copysign(sqrt(fma(alpha, alpha, nrm)), alpha);
      ti = (beta - alpha) / beta;
      sc = 1.0 / (alpha - beta);
    }
    // the vector the tiles multiply by: the row itself with x[o+1] replaced
    // by alpha - beta, that is v_o / sc
    const double x1 = alpha - beta;
    // reflector o-1 into its row, which no CTA reads any more
    if (o > 0 && rank == o % G)
      for (int r = o + 1 + tid; r < n; r += NT) __stcg(A + (size_t)(o - 1) * n + r, vw[r].x);
    if (rank == 0 && tid == 0) {
      e[o] = beta;       // for o = n-2 this is the (n-1, n-2) element
      tau[o] = ti;
      if (!next) {
        const double2 t = vw[n - 1];
        d[n - 1] = __ldcg(A + (size_t)n * n - 1) - 2.0 * t.x * t.y;
        e[n - 1] = 0.0;
        tau[n - 1] = 0.0;
      }
    }
    if (!next) break;
    // ---- (2) ----
    if (lane < kUnitRows) {
      const int r = rb0 * kUnitRows + lane;
      xfirst[lane] = r == lo ? x1 : xn[r];
    }
    __syncwarp();
    while (u < uend) {
      // one row block: its sums stay in registers, the columns' sums are added
      // to the warp's partial products unit by unit
      const int r0 = rb * kUnitRows;
      const int stop = min(uend, u + J - jb);
      const double* xrow = rb == rb0 ? xfirst : xn + r0;
      double sum[kUnitRows];
#pragma unroll
      for (int i = 0; i < kUnitRows; ++i) sum[i] = 0.0;
      while (true) {
        const int c0 = jb * kUnitCols;
        double2 vwc[2];
        double xc[2], col[2] = {0.0, 0.0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = c0 + lane + 32 * h;
          const bool ok = c < n && c >= lo;
          vwc[h] = ok ? vw[c] : make_double2(0.0, 0.0);
          xc[h] = ok ? (c == lo ? x1 : xn[c]) : 0.0;
        }
        apply_unit(row, n, live, cok, vw + r0, r0 >= c0 ? xzero : xrow, vwc, xc, a0, sum, col);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = c0 + lane + 32 * h;
          if (c < n && c >= lo) pw[c] += col[h];
        }
        ++u;
        ++jb;
        if (u >= stop) break;
        row += kUnitCols;
        cok[0] = jb * kUnitCols + lane < n;
        cok[1] = jb * kUnitCols + lane + 32 < n;
        load_unit(row, n, live, cok, a0);
      }
      const double t = reduce_rows(sum, lane);
      __syncwarp();   // the columns' sums went through other lanes
      if (lane < kUnitRows && ((live >> lane) & 1u)) pw[r0 + lane] += t;
      __syncwarp();
      ++rb;
      jb = rb / kPer;
      if (u < uend) {
        live = rows(rb);
        row = A + (size_t)rb * kUnitRows * n + jb * kUnitCols + lane;
        cok[0] = jb * kUnitCols + lane < n;
        cok[1] = jb * kUnitCols + lane + 32 < n;
        load_unit(row, n, live, cok, a0);
      }
    }
    __syncthreads();
    // ---- (3) ----
    // the CTA's sum of a row goes to the CTA that adds that row's parts
    // (blocks of 32 rows in turn), which sends the total to every CTA
    for (int r = (lo & ~31) + tid; r < n; r += NT) {
      if (r < lo) continue;
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        t += priv[w * np + r];
        priv[w * np + r] = 0.0;
      }
      const int blk = r >> 5;
      *cluster.map_shared_rank(recv + rank * slice + (blk / G) * 32 + (r & 31), blk % G) = t;
    }
    cluster.sync();
    {
      double dot = 0.0;
      // warps in turn take (block of this CTA, destination) pairs
      const int nb32 = (n + 31) >> 5, b0 = lo >> 5;
      const int q0 = b0 / G + (rank < b0 % G ? 1 : 0);          // this CTA's first live block
      const int q1 = nb32 / G + (rank < nb32 % G ? 1 : 0);
      for (int t = warp; t < (q1 - q0) * G; t += NW) {
        const int q = q0 + t / G, to = t % G;
        const int r = (q * G + rank) * 32 + lane;
        if (r >= lo && r < n) {
          double v[G], sum = 0.0;
#pragma unroll
          for (int k = 0; k < G; ++k) v[k] = recv[k * slice + q * 32 + lane];
#pragma unroll
          for (int k = 0; k < G; ++k) sum += v[k];
          *cluster.map_shared_rank(p + r, to) = sum;
          if (to == 0) dot = fma(sum, r == lo ? x1 : xn[r], dot);
        }
      }
      dot = warp_sum(dot);
      if (lane < G) *cluster.map_shared_rank(dots + rank * NW + warp, lane) = dot;
    }
    taup = ti;
    scp = sc;
    cluster.sync();
  }
  // no CTA leaves while others may still write to its shared memory
  cluster.sync();
}

template <int G, int NW>
size_t large_bytes(int n) {
  return ((size_t)(4 + NW) * padded(n) + G * slice_rows<G>(n) + (NW + 1) * kUnitRows) * sizeof(double);
}

// Launch configuration of one kernel instance (attr must outlive it).
template <int G, int NW>
cudaLaunchConfig_t config(cudaLaunchAttribute* attr, int count, size_t smem, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G * count, 1, 1);
  cfg.blockDim = dim3(32 * NW, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = G;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <int G, int NW>
void launch_cfg(const EigArgs& g, const int32_t* list, int count, int max_n, cudaStream_t stream) {
  allow_max_dynamic_smem(k_tridiag_large<G, NW>);
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = config<G, NW>(attr, count, large_bytes<G, NW>(max_n), stream);
  cudaLaunchKernelEx(&cfg, k_tridiag_large<G, NW>, g, list);
}

// Clusters of 16 CTAs (more than the portable eight) that the device runs at
// once, at the largest shared memory; 0 where it does not take them.
template <int NW>
int wide_clusters() {
  static std::mutex mu;
  static std::map<int, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  const size_t cap = allow_max_dynamic_smem(k_tridiag_large<16, NW>);
  int active = 0;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = config<16, NW>(attr, 1, cap, nullptr);
  if (cudaFuncSetAttribute(k_tridiag_large<16, NW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&active, k_tridiag_large<16, NW>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    active = 0;
  }
  known.emplace(dev, active);
  return active;
}

}  // namespace

// Each shape against its own limit: the static shared memory beside the
// vectors grows with G (16 CTAs leave 512 bytes less than eight).
template <int G, int NW>
static bool fits(int n) { return large_bytes<G, NW>(n) <= allow_max_dynamic_smem(k_tridiag_large<G, NW>); }

// Largest system (the vectors and the warps' partial products of four warps
// fill a CTA's shared memory).
bool tridiag_large_fits(int max_n) { return fits<8, 4>(max_n); }

// Systems run side by side, a cluster of eight CTAs each, two CTAs an SM (the
// vectors of up to 1090 orbitals leave room for two).
static int clusters_at_once() {
  static std::mutex mu;
  static std::map<int, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  allow_max_dynamic_smem(k_tridiag_large<8, 8>);
  int active = 0;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = config<8, 8>(attr, 1, large_bytes<8, 8>(600), nullptr);
  if (cudaOccupancyMaxActiveClusters(&active, k_tridiag_large<8, 8>, &cfg) != cudaSuccess || active < 1) {
    (void)cudaGetLastError();
    active = sm_count() / 8;
  }
  known.emplace(dev, active);
  return active;
}

// Whether `count` systems of about n orbitals end sooner on clusters than one
// to an SM.  Both sides take whole waves; a wave of the single-CTA path lasts
// as long as about (n - 107) / 118 waves of clusters.  Measured, ms of the
// clusters and of the single CTAs (33 systems fit one wave of clusters, 40 do
// not; 148 fit one wave of single CTAs):
//   258: 33 systems 1.18 / 1.52, 40: 2.25 / 1.52     300: 33 1.37 / 2.43, 40 2.68 / 2.43
//   354: 64 3.70 / 3.96, 72 5.33 / 3.96              402: 64 4.59 / 5.69, 72 6.68 / 5.68
//   450: 64 5.67 / 7.81, 72 8.15 / 7.81              504: 96 9.51 / 11.3, 128 12.7 / 12.2
//   402: 149 11.4 / 11.5, 200 15.4 / 11.7            504: 149 15.6 / 23.1, 200 20.8 / 23.5
// From 600 orbitals on the clusters win at every count tried (100: 13.4 / 19.7,
// 148: 21.8 / 22.8, 200: 29.0 / 40.1): a wave of single CTAs no longer keeps
// its matrices in L2.
bool tridiag_large_pays(int n, int count) {
  if (n >= 600) return true;
  const int at_once = clusters_at_once(), sms = sm_count();
  const int waves = (count + at_once - 1) / at_once, single = (count + sms - 1) / sms;
  return 118 * waves <= (n - 107) * single;
}

void launch_tridiag_large(const EigArgs& g, const int32_t* list, int count, int max_n, cudaStream_t stream) {
  if (count == 0) return;
  // a second set of eight CTAs pays from about 500 orbitals (600: 2.90 against
  // 3.20 ms; 360: 1.44 against 1.41) while every system still gets its SMs
  if (max_n > 480 && fits<16, 8>(max_n) && count <= wide_clusters<8>())
    launch_cfg<16, 8>(g, list, count, max_n, stream);
  else if (fits<8, 8>(max_n))
    launch_cfg<8, 8>(g, list, count, max_n, stream);
  else
    launch_cfg<8, 4>(g, list, count, max_n, stream);   // above 2208 orbitals
}

}  // namespace xtb
