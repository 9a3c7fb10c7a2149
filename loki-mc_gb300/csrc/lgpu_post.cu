// lgpu_post.cu - the reference's end-of-job routines that read the EEDF, on
// the device in FP64: the EEDF-convolved rate coefficient of every MC process
// (Collision::evaluateRateCoeff, Collision.C:355-397) and the two-term swarm
// parameters (BoltzmannMC::evaluateSwarmParameters, BoltzmannMC.C:2186-2266).
//
// Built with -fmad=false: every elementwise step rounds as the reference's
// (whose build contracts nothing), so the per-node totals of the
// momentum-transfer and energy-relaxation cross sections come out bit for
// bit; the sums over cells run as fixed-order reductions, so they agree with
// the reference's to rounding.
#include "lgpu_kernels.cuh"
#include "lgpu_launch.cuh"

namespace lgpu {

namespace {

constexpr int kPostThreads = 512;
constexpr double kQeP = 1.6021766208e-19;  // C (Constant.h:7)
constexpr double kMeP = 9.10938356e-31;    // kg (Constant.h:8)

// Sum over the block in a fixed order (every thread calls it; the result on
// every thread).
__device__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();  // red[] free again
  if (lane == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += red[k];
  return s;
}

// The grid of Grid::updateMaxValue (Grid.C:44-53) as Eigen's LinSpaced lays
// it out: node i = i * step with the last node the maximum itself; cell l =
// step/2 + l * cell step with the last cell max - step/2.
struct PostGrid {
  double max, step, lo, hi, cstep;
  int nc;
  __device__ double node(int i) const { return i == nc ? max : (double)i * step; }
  __device__ double cell(int l) const { return l == nc - 1 ? hi : lo + (double)l * cstep; }
};

// Collision::interpolatedCrossSection (Collision.C:229-288) at one energy:
// linear between the bracketing raw points (largest lower point by
// bisection), zero outside the table.
__device__ double raw_at(const double* e, const double* v, int n, double x) {
  if (n < 2 || x < e[0] || x > e[n - 1]) return 0.0;
  // (x is not negative, so the bits order as integers do, negative points included, and
  // the bisection stays off the FP64 pipe)
  const long long xb = __double_as_longlong(x);
  int lo = 0, hi = n - 1;
  while (hi > lo + 1) {
    const int mid = (hi + lo) >> 1;
    if (__double_as_longlong(e[mid]) > xb) hi = mid;
    else lo = mid;
  }
  return v[lo] + (x - e[lo]) / (e[lo + 1] - e[lo]) * (v[lo + 1] - v[lo]);
}

constexpr int kPostTile = 1024;       // cells of a block of the rates at most
constexpr int kPostRateThreads = 256;
constexpr int kPostStage = 512;       // raw points of a table staged in shared memory (longer ones stay global)
constexpr int kPostCells = 32;        // cells per block of the parameter sums
constexpr int kPostSums = 13;

__device__ __forceinline__ PostGrid post_grid(const EedfPostArgs& a) {
  PostGrid g;
  g.nc = a.nc;
  g.max = a.max_energy;
  g.step = a.max_energy / a.nc;
  g.lo = g.step / 2.0;
  g.hi = a.max_energy - g.step / 2.0;
  g.cstep = a.nc > 1 ? (g.hi - g.lo) / (a.nc - 1) : 0.0;
  return g;
}

// The EEDFs normalised from histogram sums (BoltzmannMC.C:1580: f = h /
// (sqrt(cell) sum(h) step)), one block per EEDF.
__global__ void __launch_bounds__(kPostThreads) k_post_normalise(EedfPostArgs a, double* out) {
  __shared__ double red[kPostThreads / 32];
  next_may_start();
  const PostGrid g = post_grid(a);
  const double* h = a.eeh + (size_t)blockIdx.x * a.nc;
  double* f = out + (size_t)blockIdx.x * a.nc;
  double s = 0.0;
  for (int l = threadIdx.x; l < a.nc; l += blockDim.x) s += h[l];
  const double norm = block_sum(s, red);
  for (int l = threadIdx.x; l < a.nc; l += blockDim.x) f[l] = h[l] / (sqrt(g.cell(l)) * norm * g.step);
}

// a table in shared memory when it fits (the bisection's first touches are
// then one round trip instead of one per step)
__device__ __forceinline__ void stage_table(const double*& e, const double*& v, int n, double* se, double* sv) {
  if (n > kPostStage) return;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    se[k] = e[k];
    sv[k] = v[k];
  }
  e = se;
  v = sv;
}

// EEDF-convolved rate coefficients: one block per tile of the grid's cells
// (blockIdx.x) and process (blockIdx.y). The process's cross section on the tile's
// nodes goes to shared memory and every EEDF is summed against it by a team of
// warps; the last block of a process to finish adds up the tiles' sums in their order.
// With the parameters (one EEDF) a block also writes the process's share of the
// momentum-transfer and energy-relaxation totals at its nodes, which k_post_params
// adds up in process order.
//
// Bound by FP64 issue (a warp-wide operation takes the pipe 16 cycles), so the nodes
// are spread over all SMs and the products go to the sums fused. One EEDF of 1000 cells,
// 40 processes, took 1.2 ms with one block for all, 43 us with one block per process, 19
// here; 100 EEDFs, 65 processes, 64 us before the four EEDFs side by side, 36 here.
__global__ void __launch_bounds__(kPostRateThreads) k_post_rates(EedfPostArgs a, const double* eedf, int tile) {
  constexpr int kWarps = kPostRateThreads / 32;
  next_may_start();
  __shared__ double s_e[kPostStage], s_v[kPostStage];
  __shared__ double s_me[kPostStage], s_mv[kPostStage];
  __shared__ double s_sig[kPostTile + 1];
  __shared__ double s_acc[kWarps];
  __shared__ bool s_last;
  const PostGrid g = post_grid(a);
  const int nc = a.nc, nn = nc + 1, p = blockIdx.y, tiles = gridDim.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const bool super = a.kind[p] == 2;
  // a superelastic copy convolves the forward collision's cross section with
  // the EEDF shifted by the threshold (Collision.C:390)
  const int f = super ? p - 1 : p;
  const double thr = a.thr[p], fthr = a.thr[f], dens = a.dens[p];
  const bool elastic = a.kind[f] == 0;
  const int lmin = (int)floor(thr / g.step), shift = super ? lmin : 0;
  const int ni = a.int_len[f];
  const double *ie = a.raw_ie + a.int_off[f], *iv = a.raw_iv + a.int_off[f];
  const bool shares = !a.rates_only;  // one EEDF
  // a copy's own tables (its shares) are the forward collision's, given again
  const int nm = a.mom_len[p], no = a.int_len[p];
  const double *me = a.raw_me + a.mom_off[p], *mv = a.raw_mv + a.mom_off[p];
  const double *oe = a.raw_ie + a.int_off[p], *ov = a.raw_iv + a.int_off[p];
  stage_table(ie, iv, ni, s_e, s_v);
  if (shares) stage_table(me, mv, nm, s_me, s_mv);
  wait_for_previous();  // the normalisation, if there is one
  __syncthreads();
  const int c0 = blockIdx.x * tile, cells = min(tile, nc - c0);
  for (int j = threadIdx.x; j <= cells; j += blockDim.x) {
    const int i = c0 + j;
    const double x = g.node(i);
    // on the nodes: every one for elastic collisions, from the first above the
    // threshold otherwise (Collision.C:221-228)
    const double s_int = (elastic || x > fthr) ? raw_at(ie, iv, ni, x) : 0.0;
    s_sig[j] = s_int;
    if (!shares || (j == cells && i != nc)) continue;  // the next tile's first node writes its share
    double w_mt = 0.0, w_er = 0.0, w_erc = 0.0;
    if (super) {
      // Klein-Rosseland at the nodes (Collision.C:290-353), zero at the
      // zero-energy node (BoltzmannMC.C:2205-2217)
      if (i > 0) {
        const double y = x + thr, kr = 1.0 + thr / x;
        const double w = kr * (raw_at(oe, ov, no, y) * a.stat[p]) * dens;
        w_mt = kr * (raw_at(me, mv, nm, y) * a.stat[p]) * dens;
        w_er = w * thr / x;
        w_erc = w;
      }
    } else {
      w_mt = ((elastic || x > thr) ? raw_at(me, mv, nm, x) : 0.0) * dens;
      if (elastic) {
        w_er = 2.0 * a.mass_ratio[p] * s_int * dens;
      } else {
        const double w = s_int * dens;
        w_er = i > 0 ? w * thr / x : 0.0;
        w_erc = w;
      }
    }
    double* o = a.shares + (size_t)p * nn + i;
    o[0] = w_mt;
    o[(size_t)a.P * nn] = w_er;
    o[2 * (size_t)a.P * nn] = w_erc;
  }
  __syncthreads();
  // the tile's cells from lmin on, as weights (sig_l + sig_l+1) / 2 * cell_l in place
  double keep[(kPostTile + kPostRateThreads - 1) / kPostRateThreads];
  int m = 0;
  for (int j = threadIdx.x; j < cells; j += blockDim.x, ++m)
    keep[m] = c0 + j >= lmin ? (s_sig[j] + s_sig[j + 1]) / 2.0 * g.cell(c0 + j) : 0.0;
  __syncthreads();
  m = 0;
  for (int j = threadIdx.x; j < cells; j += blockDim.x, ++m) s_sig[j] = keep[m];
  __syncthreads();
  const int j0 = max(0, lmin - c0);
  double* part = a.parts + (size_t)p * a.n_eedf * tiles + blockIdx.x;  // [EEDF][tile]
  // warps of a team share an EEDF's cells; with fewer EEDFs than warps a team has
  // several, whose sums are added up in their order
  int team = 1;
  while (2 * team * a.n_eedf <= kWarps) team *= 2;
  const int t = wid % team;
  // a warp takes four EEDFs at a time: four chains of sums in flight, and the lanes'
  // sums of all four in six steps (each lane hands half of what it has to its partner)
  constexpr int kSide = 4;
  for (int r0 = wid / team; r0 < a.n_eedf; r0 += kSide * (kWarps / team)) {
    const int stride = kWarps / team, rows = min(kSide, (a.n_eedf - r0 + stride - 1) / stride);
    const double* fr = eedf + (size_t)r0 * nc + c0 - shift;
    const size_t dr = (size_t)stride * nc;
    double s[kSide] = {0.0, 0.0, 0.0, 0.0};
    if (rows == kSide) {
      for (int j = j0 + 32 * t + lane; j < cells; j += 32 * team) {
        const double w = s_sig[j];
#pragma unroll
        for (int q = 0; q < kSide; ++q) s[q] = __fma_rn(w, fr[q * dr + j], s[q]);
      }
    } else {
      for (int q = 0; q < rows; ++q) {
        double v = 0.0;
        for (int j = j0 + 32 * t + lane; j < cells; j += 32 * team) v = __fma_rn(s_sig[j], fr[q * dr + j], v);
        s[0] = q == 0 ? v : s[0];
        s[1] = q == 1 ? v : s[1];
        s[2] = q == 2 ? v : s[2];
      }
    }
    const bool h16 = lane & 16, h8 = lane & 8;
    const double u0 = (h16 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, h16 ? s[0] : s[2], 16);
    const double u1 = (h16 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, h16 ? s[1] : s[3], 16);
    double v = (h8 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, h8 ? u0 : u1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int q = (h16 ? 2 : 0) + (h8 ? 1 : 0);  // the EEDF that this lane's sum is of
    if ((lane & 7) == 0 && q < rows) {
      if (team > 1) s_acc[wid] = v;  // (one EEDF per team then)
      else part[(size_t)(r0 + q * stride) * tiles] = v;
    }
  }
  __syncthreads();
  if (team > 1 && threadIdx.x < a.n_eedf) {
    double s = 0.0;
    for (int w = 0; w < team; ++w) s += s_acc[threadIdx.x * team + w];
    part[(size_t)threadIdx.x * tiles] = s;
  }
  // the process's last block adds up the tiles
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.ticket[1 + p], 1u) == (unsigned)tiles - 1;
    if (s_last) a.ticket[1 + p] = 0u;  // for the next call
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  const double k = sqrt(2.0 * kQeP / kMeP) * (super ? a.stat[p] : 1.0);
  for (int r = threadIdx.x; r < a.n_eedf; r += blockDim.x) {
    const double* q = a.parts + ((size_t)p * a.n_eedf + r) * tiles;
    double s = 0.0;
#pragma unroll 4
    for (int w = 0; w < tiles; ++w) s += __ldcg(&q[w]);
    s = nc > lmin ? k * s * g.step : 0.0;
    a.rates[(size_t)r * a.P + p] = s;
    a.out[(size_t)r * a.P + p] = s;
  }
}

// The two-term swarm parameters (BoltzmannMC.C:2220-2266) from the processes'
// shares: kPostCells cells per block, one node per lane and total per warp (the
// sum over processes is in their order, as the reference's), then each block's
// sums over its cells; the last block to finish adds those up in block order.
//
// Bound by latency: the loads go out many at a time, the processes' terms of the
// total ionization and attachment on a lane each, and the roots and powers of the nodes
// while k_post_rates still runs (1000 cells, 40 processes: with the sums eight loads at
// a time and everything else behind them the whole call took 60 us, 55 now).
__global__ void __launch_bounds__(128) k_post_params(EedfPostArgs a, const double* eedf) {
  __shared__ double s_tot[3][kPostCells + 1];
  __shared__ double s_k[2];
  __shared__ double s_term[2][kMaxProcesses];
  __shared__ double s_grow[kPostCells + 1];
  __shared__ bool s_last;
  const PostGrid g = post_grid(a);
  const int nc = a.nc, nn = nc + 1, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c0 = blockIdx.x * kPostCells;
  const double factor = sqrt(2.0 * kQeP / kMeP) / 3.0;
  // what the grid alone gives
  if (wid == 0)
    for (int j = lane; j <= kPostCells; j += 32)
      s_grow[j] = c0 + j > 0 && c0 + j < nn ? 1.0 / (3.0 * factor * sqrt(g.node(c0 + j))) : 0.0;
  const int l = c0 + lane;
  const double x = l < nc ? g.node(l) : 0.0;
  double pow_x = 0.0, sqrt_x = 0.0;
  if (wid >= 2 && l >= 1 && l < nc) {
    pow_x = -2.0 / 3.0 * kQeP / kMeP * pow(x, 1.5);
    sqrt_x = sqrt(x);
  }
  wait_for_previous();
  if (wid < 3) {
    for (int j = lane; j <= kPostCells; j += 32) {
      const int i = c0 + j;
      if (i >= nn) break;
      const double* q = a.shares + (size_t)wid * a.P * nn + i;
      double s = 0.0;
#pragma unroll 32
      for (int p = 0; p < a.P; ++p) s = s + q[(size_t)p * nn];
      s_tot[wid][j] = s;
    }
  } else {
    // ionization and attachment rate coefficients of the forward collisions
    for (int p = lane; p < a.P; p += 32) {
      const int kind = a.kind[p], ion = a.ion[p];
      const double term = a.dens[p] * a.rates[p];
      s_term[0][p] = kind != 2 && ion == 1 ? term : 0.0;
      s_term[1][p] = kind != 2 && ion == 2 ? term : 0.0;
    }
    __syncwarp();
    if (lane < 2) {
      double k = 0.0;
      for (int p = 0; p < a.P; ++p) k += s_term[lane][p];
      s_k[lane] = k;
    }
  }
  __syncthreads();
  const double N = a.gas_density, w = a.omega, wc = a.omega_c;
  const double k_ion = s_k[0], k_att = s_k[1], growth = k_ion - k_att;
  auto mta = [&](int j) {  // momentum transfer plus the growth term (BoltzmannMC.C:2233-2234)
    return c0 + j == 0 ? s_tot[0][j] : s_tot[0][j] + s_grow[j] * growth;
  };
  // the warps share the sums: 0..6 and, of the mobility tensor, xx and xy on
  // one warp, zz on another
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  if (l < nc) {
    const double c = g.cell(l), f = eedf[l];
    if (wid == 0) {
      for (int q = 0; q < 3; ++q) v[q] = f * c * ((s_tot[q][lane + 1] + s_tot[q][lane]) * 0.5);
      const double den = mta(lane) + mta(lane + 1);
      v[3] = c * c * f / den;
      v[4] = c * f / den;
    }
    if (wid > 0 && l >= 1) {
      const double m = mta(lane), df = f - eedf[l - 1];
      if (wid == 1) {
        v[0] = x * x * df / m;
        v[1] = x * df / m;
      } else {
        const double aux1 = pow_x * df;
        const double fr = N * m * 3.0 * factor * sqrt_x;
        const double f2 = fr * fr;
        if (wid == 2) {
          const double aux2 = (f2 + (w - wc) * (w - wc)) * (f2 + (w + wc) * (w + wc));
          v[0] = fr * (f2 + w * w + wc * wc) / aux2 * aux1;
          v[1] = w * (f2 + w * w - wc * wc) / aux2 * aux1;
          v[2] = (f2 - w * w + wc * wc) / aux2 * aux1;
          v[3] = fr / aux2 * aux1;
        } else {
          const double aux3 = f2 + w * w;
          v[0] = fr / aux3 * aux1;
          v[1] = w / aux3 * aux1;
        }
      }
    }
  }
  // warp -> first sum and count: 0: 0-4, 1: 5-6, 2: 7-10, 3: 11-12
  const int first = wid == 0 ? 0 : wid == 1 ? 5 : wid == 2 ? 7 : 11, count = wid == 0 ? 5 : wid == 2 ? 4 : 2;
  for (int q = 0; q < count; ++q) {
    double s = v[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) a.sums[(size_t)blockIdx.x * kPostSums + first + q] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    if (s_last) *a.ticket = 0u;  // for the next call
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  __shared__ double s_sum[kPostSums];
  if (threadIdx.x < kPostSums) {
    double s = 0.0;
#pragma unroll 32
    for (unsigned b = 0; b < gridDim.x; ++b) s += __ldcg(&a.sums[(size_t)b * kPostSums + threadIdx.x]);
    s_sum[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double* s = s_sum;
    const double pre = N * 3.0 * factor * g.step;
    const double v_d = 2.0 * factor * g.step * s[4], v_m = -factor * s[6];
    double* o = a.out + a.P;
    o[0] = k_ion;
    o[1] = k_att;
    o[2] = pre * s[0];
    o[3] = pre * s[1];
    o[4] = pre * s[2];
    o[5] = 2.0 * factor * g.step * s[3];
    o[6] = -factor * s[5];
    o[7] = v_d;
    o[8] = v_m;
    o[9] = v_d / v_m;
    o[10] = N * s[7];
    o[11] = -N * s[8];
    o[12] = -N * wc * s[9];
    o[13] = N * 2.0 * w * wc * s[10];
    o[14] = N * s[11];
    o[15] = -N * s[12];
  }
}

}  // namespace

// Tiles, of 32 cells at least, so that the blocks about fill the device twice (100 EEDFs
// of 1000 cells, 65 processes: 40.5 us filling it once, 36 twice).
int eedf_post_tile(int nc, int P, int sm_count) {
  const int tiles = max(1, 2 * sm_count / max(P, 1));
  const int tile = ((nc + tiles - 1) / tiles + 31) / 32 * 32;
  return min(tile, kPostTile);
}

size_t eedf_post_sums(int nc) { return (size_t)((nc + kPostCells - 1) / kPostCells) * kPostSums; }

int launch_eedf_post(const EedfPostArgs& a, int sm_count, cudaStream_t s) {
  int n = 1;
  const double* eedf = a.eedf_in;
  if (!eedf) {
    k_post_normalise<<<a.n_eedf, kPostThreads, 0, s>>>(a, a.eedf_norm);
    eedf = a.eedf_norm;
    ++n;
  }
  const int tile = eedf_post_tile(a.nc, a.P, sm_count);
  launch_after(k_post_rates, dim3((a.nc + tile - 1) / tile, a.P), kPostRateThreads, 0, s, n > 1, a, eedf, tile);
  if (!a.rates_only) {
    launch_after(k_post_params, (a.nc + kPostCells - 1) / kPostCells, 128, 0, s, true, a, eedf);
    ++n;
  }
  return n;
}

}  // namespace lgpu
