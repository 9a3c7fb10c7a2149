// lgpu_kernels.cu - sm_103a kernels of the electron Monte Carlo path.
//
//   k_advance       free flights + collisions of every electron up to the
//                   synchronisation time (BoltzmannMC.C:617-688, 804-1280)
//   k_init          Maxwellian start ensemble (BoltzmannMC.C:491-508)
//   k_build_tables  FP64 interpolated tables -> FP32 row pairs
//                   (BoltzmannMC.C:561-615)
//   k_sample        ensemble moments and maximum energy (BoltzmannMC.C:1410-1446)
//   k_hist          EEDF / EADF / EVDF tallies (BoltzmannMC.C:1550-1571)
//   k_pop_*         population control after ionization and attachment
//                   (BoltzmannMC.C:1282-1408)
//   k_replay_*      the same device functions on given inputs (parity tests)
#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>

#include "lgpu_advance.cuh"
#include "lgpu_device.cuh"
#include "lgpu_interval_end.h"
#include "lgpu_kernels.cuh"

namespace lgpu {

namespace {

// the main pass over the ensemble
template <int MODE, int BLOCKS_PER_SM>
__global__ void __launch_bounds__(kAdvanceThreads, BLOCKS_PER_SM) k_advance(const __grid_constant__ AdvanceArgs a) {
  __shared__ AdvShared sh;
  advance_body<MODE>(a, sh);
}
// ------------------------------------------------------------------ init
__global__ void k_init(InitArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float e = 0.0f;
  if (i < a.n) {
    PhiloxStream rng;
    rng.init((uint32_t)i, 0xFFFFFFFFFFFFull, a.seed, 0x7u);
    // three normals from four uniforms (Box-Muller, MathFunctions.C:54-59)
    const float r1 = rng.oc(), r2 = rng.oc(), r3 = rng.oc(), r4 = rng.oc();
    const float aa = sqrtf(-2.0f * logf(r1));
    float sb, cb;
    sincosf(kTwoPiF * r2, &sb, &cb);
    const float3 v = make_float3(aa * cb * a.sd, aa * sb * a.sd, sqrtf(-2.0f * logf(r3)) * cosf(kTwoPiF * r4) * a.sd);
    a.state[2 * i] = make_float4(0.f, 0.f, 0.f, -1.0f);
    a.state[2 * i + 1] = make_float4(v.x, v.y, v.z, 0.0f);
    e = energy_of(v, a.half_me_over_e);
  }
  e = warp_max(e);
  if ((threadIdx.x & 31) == 0 && e > 0.0f) atomic_max_energy(a.max_energy_bits, e);
}

// --------------------------------------------------------------- tables
// Linear interpolation of the raw table (the bracketing index by bisection,
// largest i with x_i <= x clamped to n-2, then y_i + (x-x_i)/(x_{i+1}-x_i)*(y_{i+1}-y_i)),
// with explicit round-to-nearest operations so no FMA contraction happens.
// x is not negative, so that its bits order against the points' as integers do: the
// bisection stays off the FP64 pipe.
__device__ __forceinline__ double interp_raw(const double* xs, const double* ys, int n, double x) {
  const long long xb = __double_as_longlong(x);
  int lo = 0, hi = n - 1;
  while (hi > lo + 1) {
    const int mid = (hi + lo) >> 1;
    if (__double_as_longlong(__ldg(&xs[mid])) > xb) hi = mid; else lo = mid;
  }
  const double dx = __dsub_rn(xs[lo + 1], xs[lo]);
  return __dadd_rn(ys[lo], __dmul_rn(__ddiv_rn(__dsub_rn(x, xs[lo]), dx), __dsub_rn(ys[lo + 1], ys[lo])));
}

// sigma*n of process p at `energy` (a superelastic process reads its
// inelastic partner's raw table at energy + threshold)
__device__ __forceinline__ double table_value(const TableBuildArgs& a, int p, double energy) {
  if (a.is_super[p]) {
    if (energy > a.emin[p] && energy <= a.emax[p]) {
      const double thr = a.emin[p - 1];
      const double sg = interp_raw(a.raw_e + a.raw_off[p - 1], a.raw_v + a.raw_off[p - 1], a.raw_len[p - 1],
                                   __dadd_rn(energy, thr));
      return __dmul_rn(__dmul_rn(__dmul_rn(a.superw[p], __dadd_rn(1.0, __ddiv_rn(thr, energy))), sg), a.rel_dens[p]);
    }
  } else if (energy >= a.emin[p] && energy <= a.emax[p]) {
    return __dmul_rn(interp_raw(a.raw_e + a.raw_off[p], a.raw_v + a.raw_off[p], a.raw_len[p], energy), a.rel_dens[p]);
  }
  return 0.0;
}

// 32 energy rows per block, one per lane: the warps interpolate a process each for
// all rows (neighbouring energies share raw intervals, and rows below a threshold
// cost nothing), then one warp sums every lane's row over the processes in their order
// (which fixes the FP64 rounding) and all warps write FP32 row pairs.
//
// Bound by FP64 issue: a warp-wide FP64 operation takes the pipe 16 cycles whatever its
// active lanes. With the lanes on the processes of one row, a row's sum and its
// frequency ran on one lane each: 10,000 rows of 2, 40 and 65 processes took 34, 95
// and 140 us, 8, 31 and 44 here (44 ms of the 64-point sweep's 395: 64 first tables
// and 200 re-grids beside its intervals).
constexpr int kTableRows = 32, kTablePitch = kTableRows + 1;  // shared-memory pitch of a process's rows
constexpr int kTableThreads = 256, kTableThreadsAlone = 1024;  // (launch_build_tables)

constexpr int table_smem(int P) { return P * kTablePitch * (int)(sizeof(double) + sizeof(float)); }

template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_build_tables(TableBuildArgs a) {
  extern __shared__ double s_val[];  // [P][kTablePitch] sigma*n, then the FP32 cumulative sums
  const int P = a.P, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float* s_cum = reinterpret_cast<float*>(s_val + P * kTablePitch);
  const int i0 = blockIdx.x * kTableRows, rows = min(kTableRows, a.M - i0), i = i0 + lane;
  const double energy = __dmul_rn((double)i, a.step);
  for (int p = w; p < P; p += THREADS / 32)
    s_val[p * kTablePitch + lane] = lane < rows ? table_value(a, p, energy) : 0.0;
  __syncthreads();
  if (w == 0) {
    double cur = 0.0;
#pragma unroll 8
    for (int p = 0; p < P; ++p) {
      cur = __dadd_rn(cur, s_val[p * kTablePitch + lane]);
      s_cum[p * kTablePitch + lane] = (float)cur;
      if (a.cum64 && lane < rows) a.cum64[(size_t)i * P + p] = cur;
    }
    if (lane < rows) {
      const double kq = 1.6021766208e-19, km = 9.10938356e-31;
      const double nu = __dmul_rn(cur, __dmul_rn(a.N, __dsqrt_rn(__ddiv_rn(__dmul_rn(__dmul_rn(energy, 2.0), kq), km))));
      a.nu_tot[i] = nu;
      a.nu_pair[i].x = (float)nu;
      if (i > 0) a.nu_pair[i - 1].y = (float)nu;
      if (i == a.M - 1) a.nu_pair[i].y = (float)nu;
    }
  }
  __syncthreads();
  // pair (row, next row); the next block's first row completes this one's last
  for (int k = threadIdx.x; k < rows * a.stride; k += THREADS) {
    const int r = k / a.stride, p = k - r * a.stride;
    const size_t o = (size_t)(i0 + r) * a.stride + p;
    if (p >= P) {
      // row padding: a cumulative value no random number reaches, zero rate
      a.cum_pair[o] = make_float2(3.0e38f, 3.0e38f);
      a.sig_pair[o] = make_float2(0.0f, 0.0f);
      continue;
    }
    const double value = s_val[p * kTablePitch + r];
    const float vf = (float)value, cf = s_cum[p * kTablePitch + r];
    if (a.sig64) a.sig64[(size_t)(i0 + r) * P + p] = value;
    const int next = i0 + r == a.M - 1 ? r : r + 1;  // the last row pairs with itself
    if (next < rows) {
      a.sig_pair[o] = make_float2(vf, (float)s_val[p * kTablePitch + next]);
      a.cum_pair[o] = make_float2(cf, s_cum[p * kTablePitch + next]);
    } else {
      a.sig_pair[o].x = vf;
      a.cum_pair[o].x = cf;
    }
    if (r == 0 && i0 > 0) {
      a.sig_pair[o - a.stride].y = vf;
      a.cum_pair[o - a.stride].y = cf;
    }
  }
}

// Running maximum of nu_tot (block 0: a run of rows per warp; max is exact in any
// order) and the block bounds of the total frequency for
// the coarse null test (other blocks, one warp each): the largest FP32 value of rows
// [b R, (b+1) R] (row pairs cover the next row), raised by 2^-20 relative against
// the rounding of the interpolation. Tiles of 1024 rows one after the other, and one
// thread per bound in a launch of its own, took 33 + 8.6 us for 10,000 rows; this
// takes 12.
constexpr int kPrefixThreads = 1024;

__global__ void __launch_bounds__(kPrefixThreads) k_table_bounds(const double* nu_tot, double* nu_max, int M,
                                                                const float2* nu_pair, int shift, float* coarse,
                                                                int n_coarse) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (blockIdx.x > 0) {
    const int b = (blockIdx.x - 1) * (kPrefixThreads / 32) + w;
    if (b >= n_coarse) return;
    const int last = min((b + 1) << shift, M);
    float m = 0.0f;
    for (int i = (b << shift) + lane; i < last; i += 32) {
      const float2 v = nu_pair[i];
      m = fmaxf(m, fmaxf(v.x, v.y));
    }
    m = warp_max(m);
    if (lane == 0) coarse[b] = m * (1.0f + 9.5367431640625e-7f);
    return;
  }
  // each warp has a run of rows of its own, 32 at a time; the frequencies' bits are
  // compared as integers, off the FP64 pipe (from 0 up, and no number never the
  // larger one, as fmax has it)
  __shared__ long long s_w[kPrefixThreads / 32];
  auto key = [&](int i) {
    const long long k = i < M ? __double_as_longlong(nu_tot[i]) : 0;
    return k <= 0x7ff0000000000000ll ? max(k, 0ll) : 0ll;
  };
  const int run = (M + kPrefixThreads - 1) / kPrefixThreads * 32;
  const int first = (int)min((long long)w * run, (long long)M), last = (int)min((long long)first + run, (long long)M);
  long long v = 0;
#pragma unroll 4
  for (int i = first + lane; i < last; i += 32) v = max(v, key(i));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) s_w[w] = v;
  __syncthreads();
  long long before = lane < w ? s_w[lane] : 0;  // the rows of the warps before this one
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before = max(before, __shfl_xor_sync(0xffffffffu, before, o));
#pragma unroll 4
  for (int i0 = first; i0 < last; i0 += 32) {
    v = key(i0 + lane);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v = max(v, u);
    }
    v = max(v, before);
    if (i0 + lane < last) nu_max[i0 + lane] = __longlong_as_double(v);
    before = __shfl_sync(0xffffffffu, v, 31);
  }
}

// ---------------------------------------------------------------- sample
constexpr int kSampleThreads = 512;        // blocks that count without shared EADF and EVDF cells
constexpr int kSampleSharedThreads = 1024;  // and with them: one block per SM
// Their shared memory: EEDF (1000 cells), the slower rows of the EVDF and the lower
// rows of the EADF. No more than this: the loads in flight live in what is left for
// L1 (the EADF pass this replaces took 193 us per sweep interval with 224 KB of
// counts and 160 with 195).
constexpr int kSampleSmem = 124 * 1024;
constexpr int kSampleSmemV = 56 * 1024;    // of it, at most, the EVDF's

// Moment sums of electrons begin, begin+step, ... < end into a.moments: per
// thread in FP32 (a handful of electrons each), FP64 from the warp reduction on.
// Every thread of the block calls this; s_m is the block's scratch.
struct NoExtra {
  __device__ __forceinline__ void operator()(float4) const {}
};

// `extra` sees every electron's (vx, vy, vz, flag) in the same pass (the distributions
// are counted with it)
template <class Extra = NoExtra>
__device__ __forceinline__ void sample_range(const SampleArgs& a, int begin, int end, int step,
                                             double (*s_m)[kMoments], Extra extra = Extra()) {
  float m[kMoments];
#pragma unroll
  for (int k = 0; k < kMoments; ++k) m[k] = 0.0f;
  float e_max = 0.0f;
  auto add = [&](float4 A, float4 B) {
    extra(B);
    const float e = energy_of(make_float3(B.x, B.y, B.z), a.half_me_over_e);
    e_max = fmaxf(e_max, e);
    const float x = A.x, y = A.y, z = A.z, vx = B.x, vy = B.y, vz = B.z;
    m[0] += e;
    m[1] += x; m[2] += y; m[3] += z;
    m[4] += vx; m[5] += vy; m[6] += vz;
    m[7] += x * x; m[8] += x * y; m[9] += x * z; m[10] += y * y; m[11] += y * z; m[12] += z * z;
    m[13] += x * vx; m[14] += x * vy; m[15] += x * vz;
    m[16] += y * vx; m[17] += y * vy; m[18] += y * vz;
    m[19] += z * vx; m[20] += z * vy; m[21] += z * vz;
  };
  // four electrons' loads in flight before their sums (memory-level parallelism)
  int i = begin;
  for (; i + 3 * step < end; i += 4 * step) {
    float4 A[4], B[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) load_record(a.state + 2 * (i + u * step), A[u], B[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) add(A[u], B[u]);
  }
  for (; i < end; i += step) {
    float4 A, B;
    load_record(a.state + 2 * i, A, B);
    add(A, B);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // FP32 tree reduction inside the warp (32 partials), FP64 across warps and blocks
#pragma unroll
  for (int k = 0; k < kMoments; ++k) {
    float w = m[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane == 0) s_m[wid][k] = (double)w;
  }
  e_max = warp_max(e_max);
  if (lane == 0 && e_max > 0.0f) atomic_max_energy(a.max_energy_bits, e_max);
  __syncthreads();
  if (threadIdx.x < kMoments) {
    double sum = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += s_m[w][threadIdx.x];
    atomicAdd(&a.moments[threadIdx.x], sum);
  }
}

// ------------------------------------------------------------- histograms
// The tallies of one sample in two passes over the electrons' velocities,
// each in blocks of up to kHistChunk electrons that count in shared memory and
// then add one atomic per occupied cell to the FP64 tallies:
//   pass A: EEDF counts (32-bit) and EADF counts (16-bit, two per word),
//   pass B: EVDF counts (16-bit, two per word), cylindrical conditions only.
// A block's chunk is below 2^16 electrons, so no 16-bit count can carry into
// its neighbour. A condition whose grid is larger than the block's shared
// memory counts that tally with global atomics instead.
constexpr int kHistChunk = kBatchHistChunk;  // below 2^16: 16-bit counts cannot carry
constexpr int kHistAThreads = 1024;
constexpr int kHistBThreads = 512;
constexpr int kHistASmem = 195 * 1024;  // one block per SM
constexpr int kHistBSmem = 96 * 1024;   // two blocks per SM

__device__ __forceinline__ float radial_speed(float v2xy) { return v2xy > 0.0f ? v2xy * rsqrtf(v2xy) : 0.0f; }

__device__ __forceinline__ void velocity_cell(const HistArgs& a, float4 B, int& rx, int& ry) {
  rx = (int)(radial_speed(__fmaf_rn(B.y, B.y, __fmul_rn(B.x, B.x))) * a.inv_rad_step);
  ry = (int)((B.z + a.max_speed) * a.inv_ax_step);
}

__device__ __forceinline__ void hist_cells(const HistArgs& a, float4 B, int& c, int& cy, int& rx, int& ry) {
  // MathFunctions.C:61-81 (energy) and 106-127 (energy x cos, radial x axial velocity)
  const float v2xy = __fmaf_rn(B.y, B.y, __fmul_rn(B.x, B.x));
  const float v2 = __fmaf_rn(B.z, B.z, v2xy);
  const float e = __fmul_rn(v2, a.half_me_over_e);  // energy_of's rounding
  c = (int)(e * a.inv_e_step);
  cy = rx = ry = -1;
  if (a.cylindrical) {
    // cos and radial speed from the hardware reciprocal square root: a cell
    // edge moves by a few 1e-7 relative, far below the statistical resolution
    // of any cell (a zero speed has no angle and stays outside the cos cells)
    const float cosang = v2 > 0.0f ? B.z * rsqrtf(v2) : 2.0f;
    cy = (int)((cosang + 1.0f) * (0.5f * (float)a.n_cos));
    velocity_cell(a, B, rx, ry);
  }
}

// the calling block, for end_interval
struct ThisBlock {
  __device__ __forceinline__ int thread() const { return (int)threadIdx.x; }
  __device__ __forceinline__ int threads() const { return (int)blockDim.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  template <class T>
  __device__ __forceinline__ T load(const T* p) const { return __ldcg(p); }
};

__device__ __forceinline__ void end_plain_interval(const SampleArgs& a, bool sampled) {
  end_interval(ThisBlock(), a.plain->ctl, a.plain->dist, a.plain->chain, a.sc, a.n, a.out->sc, 1, &a.out->done, nullptr,
               sampled);
}

__global__ void k_interval_end(SampleArgs a) {
  next_may_start();
  wait_for_previous();
  end_plain_interval(a, false);
}

// The cells a block counts in shared memory (16-bit, two per word: a block sees fewer
// than 2^16 electrons before it adds them up): the EADF's energy rows and the EVDF's
// radial rows from zero up, as many as fit. The grids reach beyond the fastest
// electron by a fifth, so that the rows left out hold the last per mille of the
// electrons; those are added to the FP64 tallies one by one.
struct SharedCells {
  int a_rows, v_rows;
};
__host__ __device__ __forceinline__ SharedCells shared_cells(int n_e, int n_cos, int n_rad, int n_ax) {
  SharedCells c;
  c.v_rows = min(n_rad, kSampleSmemV / 2 / max(n_ax, 1));
  const long long left = kSampleSmem - 4ll * n_e - 4 * (((long long)c.v_rows * n_ax + 1) / 2) - 8;
  c.a_rows = (int)min((long long)n_e, max(left, 0ll) / 2 / max(n_cos, 1));
  return c;
}

// Moments and distributions of electrons first, first + step, ... < end in one
// read: EEDF counts in shared memory (one FP64 addition per occupied cell and
// block), EADF and EVDF counts there too (shared) or straight to the FP64 tallies,
// where few electrons of a block share a cell. Every thread of the block calls this.
//
// Straight counts are bound by the FP64 additions at L2 (1.1e11/s at best, faster than
// 32-bit ones to the same cells, and about 7e10/s on the swarms' own cells), shared
// ones by the read of the ensemble.
__device__ __forceinline__ void sample_counting(const SampleArgs& a, const HistArgs& h, bool shared, int first,
                                                int end, int step, double (*s_m)[kMoments], unsigned int* sm_dist) {
  const int nE = h.n_e_cells;
  const SharedCells sc = shared && h.cylindrical ? shared_cells(nE, h.n_cos, h.n_rad, h.n_ax) : SharedCells{0, 0};
  const int nA = sc.a_rows * h.n_cos, nV = sc.v_rows * h.n_ax, nAw = (nA + 1) >> 1, nVw = (nV + 1) >> 1;
  unsigned int* hE = sm_dist;
  unsigned int* hA = hE + nE;
  unsigned int* hV = hA + nAw;
  for (int c = threadIdx.x; c < nE + nAw + nVw; c += blockDim.x) sm_dist[c] = 0u;
  __syncthreads();
  // (an EEDF cell whose EADF row is shared is that row's sum and what is counted
  // apart: electrons outside the cos cells, cos rounding to 1 or zero speed)
  auto count = [&](float4 B) {
    int c, cy, rx, ry;
    hist_cells(h, B, c, cy, rx, ry);
    if (c >= 0 && c < nE) {
      const bool angle = cy >= 0 && cy < h.n_cos;
      const int idx = c * h.n_cos + cy;
      if (angle && idx < nA) {
        atomicAdd(&hA[idx >> 1], 1u << ((idx & 1) << 4));
      } else {
        atomicAdd(&hE[c], 1u);
        if (angle) atomicAdd(&h.eadf[idx], 1.0);
      }
    }
    if (rx >= 0 && rx < h.n_rad && ry >= 0 && ry < h.n_ax) {
      const int idx = rx * h.n_ax + ry;
      if (idx < nV) atomicAdd(&hV[idx >> 1], 1u << ((idx & 1) << 4));
      else atomicAdd(&h.evdf[idx], 1.0);
    }
  };
  sample_range(a, first, end, step, s_m, count);  // ends behind a block barrier
  for (int c = threadIdx.x; c < nE; c += blockDim.x) {
    unsigned int k = hE[c];
    if (c < sc.a_rows)
      for (int q = 0; q < h.n_cos; ++q) {
        const int idx = c * h.n_cos + q;
        k += (hA[idx >> 1] >> ((idx & 1) << 4)) & 0xFFFFu;
      }
    if (!k) continue;
    atomicAdd(&h.eedf[c], (double)k);
    if (h.eedf_periodic_row) atomicAdd(&h.eedf_periodic_row[c], (double)k);
  }
  for (int w = threadIdx.x; w < nAw + nVw; w += blockDim.x) {
    const unsigned int k = hA[w];
    if (!k) continue;
    double* cell = w < nAw ? h.eadf + 2 * w : h.evdf + 2 * (w - nAw);
    if (k & 0xFFFFu) atomicAdd(&cell[0], (double)(k & 0xFFFFu));
    if (k >> 16) atomicAdd(&cell[1], (double)(k >> 16));
  }
}

// The sample of one condition: the moments and, when the interval's DistCtl says
// so, the distributions. Separate passes over the electrons in 65535-electron chunks,
// which this replaces up to kDistInSample electrons, left most SMs idle: moments +
// EEDF/EADF + EVDF of 1e6 electrons 16 + 49 + 91 -> 35 us, of 4e6 28 + 54 + 93 -> 65,
// of 10,000 5 + 12 + 14.5 -> 7.
template <bool SHARED>
__global__ void __launch_bounds__(SHARED ? kSampleSharedThreads : kSampleThreads, SHARED ? 1 : 2)
    k_sample(SampleArgs a) {
  __shared__ double s_m[(SHARED ? kSampleSharedThreads : kSampleThreads) / 32][kMoments];
  __shared__ bool s_last;
  extern __shared__ unsigned int sm_dist[];
  next_may_start();
  wait_for_previous();
  if (a.plain && !a.plain->ctl.go) return;  // the chain of intervals has stopped
  const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  const bool counts = a.plain && a.plain->dist.on &&
                      __uint_as_float(a.sc->max_energy_bits) <= a.plain->dist.e_bound;
  if (counts) sample_counting(a, a.plain->dist.h, SHARED, first, a.n, step, s_m, sm_dist);
  else sample_range(a, first, a.n, step, s_m);
  if (!a.plain) return;
  // the last block ends the interval
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.plain->ticket, 1u) == gridDim.x - 1;
    if (s_last) a.plain->ticket = 0u;
    __threadfence();
  }
  __syncthreads();
  if (s_last) end_plain_interval(a, true);
}

// Below this many electrons a chunk counts EADF and EVDF with global atomics:
// clearing and scanning the whole shared-memory grid would cost more.
constexpr int kHistSharedMin = 16384;

// pass A over electrons [first, last) of one condition. Shared memory holds the
// EEDF counts and as many of the EADF's rows as fit (SHARED rows), the rest, at the
// top of the energy grid where hardly an electron is, goes to global atomics.
__device__ __forceinline__ void hist_chunk_a(const HistArgs& a, int first, int last, unsigned int* sm, int sm_words) {
  const int nE = a.n_e_cells;
  const int nA = a.cylindrical ? nE * a.n_cos : 0;
  const bool a_shared = a.cylindrical && last - first >= kHistSharedMin && nE < sm_words;
  // cells of whole energy rows in shared memory
  const int nS = a_shared ? min(nE, (int)(2ll * (sm_words - nE) / a.n_cos)) * a.n_cos : 0;
  const int nSw = (nS + 1) >> 1;
  unsigned int* hE = sm;
  unsigned int* hA = sm + nE;
  for (int w = threadIdx.x; w < nE + nSw; w += blockDim.x) sm[w] = 0u;
  __syncthreads();
  // An EEDF count of a cell whose EADF row is in shared memory is that row's sum,
  // so only electrons outside the cos cells (cos rounding to 1, zero speed) and
  // the rows left out are counted into hE: one shared-memory atomic per electron.
  auto bin = [&](float4 B) {
    int c, cy, rx, ry;
    hist_cells(a, B, c, cy, rx, ry);
    if (c >= 0 && c < nE) {
      if (a.cylindrical && cy < a.n_cos && cy >= 0) {
        const int idx = c * a.n_cos + cy;
        if (idx < nS) {
          atomicAdd(&hA[idx >> 1], 1u << ((idx & 1) << 4));
        } else {
          atomicAdd(&hE[c], 1u);
          atomicAdd(&a.eadf[idx], 1.0);
        }
      } else {
        atomicAdd(&hE[c], 1u);
      }
    }
  };
  // four electrons' loads in flight per thread before their counts; each
  // warp bulk-prefetches into L2 its 128 records of the block's pass two
  // rounds ahead
  const int st = blockDim.x;
  auto prefetch_round = [&](int base) {
    const int e0 = base + (int)(threadIdx.x >> 5) * 128;
    if ((threadIdx.x & 31) == 0 && e0 < last) prefetch_l2(a.state + 2 * e0, (uint32_t)min(128, last - e0) * 32u);
  };
  prefetch_round(first);
  prefetch_round(first + 4 * st);
  int i = first + threadIdx.x;
  for (; i + 3 * st < last; i += 4 * st) {
    prefetch_round(i - (int)threadIdx.x + 8 * st);
    const float4 B0 = a.state[2 * i + 1], B1 = a.state[2 * (i + st) + 1];
    const float4 B2 = a.state[2 * (i + 2 * st) + 1], B3 = a.state[2 * (i + 3 * st) + 1];
    bin(B0);
    bin(B1);
    bin(B2);
    bin(B3);
  }
  for (; i < last; i += st) bin(a.state[2 * i + 1]);
  __syncthreads();
  for (int c = threadIdx.x; c < nE; c += blockDim.x) {
    unsigned int h = hE[c];
    if (c * a.n_cos < nS) {
      for (int k = 0; k < a.n_cos; ++k) {
        const int idx = c * a.n_cos + k;
        h += (hA[idx >> 1] >> ((idx & 1) << 4)) & 0xFFFFu;
      }
    }
    if (h) {
      atomicAdd(&a.eedf[c], (double)h);
      if (a.eedf_periodic_row) atomicAdd(&a.eedf_periodic_row[c], (double)h);
    }
  }
  for (int w = threadIdx.x; w < nSw; w += blockDim.x) {
    const unsigned int h = hA[w];
    if (h & 0xFFFFu) atomicAdd(&a.eadf[2 * w], (double)(h & 0xFFFFu));
    if ((h >> 16) && 2 * w + 1 < nA) atomicAdd(&a.eadf[2 * w + 1], (double)(h >> 16));
  }
  __syncthreads();
}

// pass B over electrons [first, last) of one cylindrical condition
__device__ __forceinline__ void hist_chunk_b(const HistArgs& a, int first, int last, unsigned int* sm, int sm_words) {
  const int nV = a.n_rad * a.n_ax;
  const int nVw = (nV + 1) >> 1;
  const bool v_shared = last - first >= kHistSharedMin && nVw <= sm_words;
  if (v_shared)
    for (int w = threadIdx.x; w < nVw; w += blockDim.x) sm[w] = 0u;
  __syncthreads();
  for (int i = first + threadIdx.x; i < last; i += blockDim.x) {
    int c, cy, rx, ry;
    hist_cells(a, a.state[2 * i + 1], c, cy, rx, ry);
    if (rx < a.n_rad && rx >= 0 && ry < a.n_ax && ry >= 0) {
      const int idx = rx * a.n_ax + ry;
      if (v_shared) atomicAdd(&sm[idx >> 1], 1u << ((idx & 1) << 4));
      else atomicAdd(&a.evdf[idx], 1.0);
    }
  }
  __syncthreads();
  if (v_shared) {
    for (int w = threadIdx.x; w < nVw; w += blockDim.x) {
      const unsigned int h = sm[w];
      if (h & 0xFFFFu) atomicAdd(&a.evdf[2 * w], (double)(h & 0xFFFFu));
      if ((h >> 16) && 2 * w + 1 < nV) atomicAdd(&a.evdf[2 * w + 1], (double)(h >> 16));
    }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kHistAThreads) k_hist_a(HistArgs a) {
  extern __shared__ unsigned int sm_hist[];
  const int chunks = (a.n + kHistChunk - 1) / kHistChunk;
  for (int c = blockIdx.x; c < chunks; c += gridDim.x)
    hist_chunk_a(a, c * kHistChunk, min(a.n, (c + 1) * kHistChunk), sm_hist, kHistASmem / 4);
}

__global__ void __launch_bounds__(kHistBThreads) k_hist_b(HistArgs a) {
  extern __shared__ unsigned int sm_hist[];
  const int chunks = (a.n + kHistChunk - 1) / kHistChunk;
  for (int c = blockIdx.x; c < chunks; c += gridDim.x)
    hist_chunk_b(a, c * kHistChunk, min(a.n, (c + 1) * kHistChunk), sm_hist, kHistBSmem / 4);
}

// One block per column on the energy grid: the EEDF, each angle's EADF column, each
// phase's EEDF. A cell of the new grid adds, in their order, the shares of the old
// cells that reach into it (an old cell is narrower than a new one and reaches into
// two at most). As in the reference, the per-phase sums are not cleared first and
// take every old cell once per phase (BoltzmannMC.C:1523-1541).
//
// Bound by the FP64 divisions that place an old cell: done once per cell, to shared
// memory, 1000 cells and 100 angles take 19 us, and took 75 with every new cell
// placing the old ones about it again. On the host, between two copies of all tallies
// and with every per-phase cell added once per phase one by one, re-binning was most of
// the 311 us of host work per interval of 32 conditions in crossed B and AC fields (64
// phases); 28 are left.
constexpr int kRebinThreads = 256;
// old value, its share of the lower new cell, that cell (twice, plus one if the old cell
// reaches into the next)
constexpr int kRebinCell = 2 * sizeof(double) + sizeof(int);

__global__ void __launch_bounds__(kRebinThreads) k_rebin(RebinArgs a) {
  extern __shared__ double rebin_old[];
  const int col = blockIdx.x, nE = a.n_e;
  double* old = rebin_old;
  double* share = old + nE;
  int* place = reinterpret_cast<int*>(share + nE);
  const bool phase = col > a.n_cos;
  double* v = col == 0 ? a.eedf : phase ? a.eedf_per + (size_t)(col - 1 - a.n_cos) * nE : a.eadf + (col - 1);
  const int stride = col == 0 || phase ? 1 : a.n_cos;
  for (int o = threadIdx.x; o < nE; o += blockDim.x) {
    old[o] = v[(size_t)o * stride];
    const double lo = o * a.old_step, hi = o + 1 == nE ? a.old_max : (o + 1) * a.old_step;
    const int nl = (int)(lo / a.step), nr = (int)(hi / a.step);
    share[o] = nl == nr ? 1.0 : (nr * a.step - lo) / a.old_step;
    place[o] = 2 * nl + (nl != nr);
  }
  __syncthreads();
  const double ratio = a.step / a.old_step;
  for (int c = threadIdx.x; c < nE; c += blockDim.x) {
    double s = 0.0;
    const int first = max(0, (int)fmin(c * ratio, (double)nE) - 2), last = min(nE - 1, (int)fmin((c + 1) * ratio, (double)nE) + 2);
    for (int o = first; o <= last; ++o) {
      const int at = place[o];
      if (at >> 1 == c) s += share[o] * old[o];
      else if (at == 2 * c - 1) s += (1.0 - share[o]) * old[o];
    }
    v[(size_t)c * stride] = phase ? old[c] + a.n_phases * s : s;
  }
}

// ------------------------------------------------------- population control
__device__ __forceinline__ uint32_t pop_word(uint32_t idx, uint64_t interval, uint64_t seed, uint32_t salt,
                                             uint32_t draw) {
  Philox ph;
  ph.ctr = make_uint4(idx, (uint32_t)interval, (uint32_t)(interval >> 32) ^ (salt << 16), 0x80000000u | draw);
  ph.key = make_uint2((uint32_t)(seed ^ 0xA5A5A5A5u), (uint32_t)(seed >> 32));
  return ph.next().x;
}

// uniform integer in [0, n) from a 32-bit word (n < 2^31)
__device__ __forceinline__ int uniform_index(uint32_t w, int n) {
  return (int)(((unsigned long long)w * (unsigned long long)n) >> 32);
}

// adds a per-thread energy to the growth accumulator with one atomic per warp
__device__ __forceinline__ void add_growth(double* growth, double e) {
  cg::coalesced_group g = cg::coalesced_threads();
  const double tot = cg::reduce(g, e, cg::plus<double>());
  if (g.thread_rank() == 0) atomicAdd(growth, tot);
}

__device__ __forceinline__ float energy4(float4 B, float hme) { return energy_of(make_float3(B.x, B.y, B.z), hme); }

// Population control (BoltzmannMC.C:1282-1408), when all electrons and
// secondaries are at the synchronisation time (every listed secondary is alive:
// one that attached was not listed). The secondaries that a condition's warps could
// not queue come first: there seldom are any, and then one block pushes them and
// does the condition's first phase. Three launches, each a grid over the items
// of one or many slots. With n_att attached slots and n_sec secondaries:
//  (a) the first min(n_att, n_sec) attached slots take the last secondaries
//      (:1344-1359); slots left attached are marked in the claim bitmap, so that no
//      clone is made from another clone; or, when secondaries are left over, a
//      uniformly random subset of their number m is drawn from the pool of N slots
//      + m unplaced secondaries - the outcome of the reference's sequential uniform
//      removal (:1379-1407) - by claiming pool bits. No item depends on another:
//      marks and draws never meet in one interval, and a slot drawn while it takes
//      its secondary is read in the next phase;
//  (b) the slots left attached clone a random non-attached electron, whose energy
//      enters the growth term (:1360-1376); or the removed ensemble slots and the
//      unremoved secondaries are listed, removed energies leave the growth term;
//  (c) the listed secondaries move into the removed slots; all marks are cleared,
//      so the bitmap is zero again.
//
// Bound by latency: a handful of dependent loads per launch on few items. Listing,
// filling, drawing, sorting and placing in a launch each, after another for the
// spilled secondaries, took 25 us per interval for 1e6 electrons alone and 39 for
// 32 conditions of 10,000-30,000; these three take 15 and 24. One launch of a
// cluster per condition with a barrier between the phases took 14 and 26, but 7 %
// more of the whole sweep: its largest conditions need more than a cluster's threads.
constexpr int kPopThreads = 256;
constexpr int kPopBlocks = 64;           // blocks, single condition
constexpr int kPopBlocksPerSM = 2;       // blocks per SM, batches

// one condition, arguments by value
struct PopOne {
  PopArgs a;
  AdvanceArgs adv;
  __device__ int count() const { return 1; }
  __device__ const AdvanceArgs* advance(int) const { return &adv; }
  __device__ const PopArgs* get(int s) const { return s == 0 ? &a : nullptr; }
};
// the slots of a batch that ionize or attach
struct PopBatch {
  const BatchHeader* hdr;
  const BatchSlot* slots;
  __device__ int count() const { return hdr->n_slots; }
  __device__ const AdvanceArgs* advance(int s) const { return &slots[s].adv; }
  __device__ const PopArgs* get(int s) const {
    return (s < hdr->n_slots && (slots[s].flags & kSlotIonAtt)) ? &slots[s].pop : nullptr;
  }
};

__device__ __forceinline__ int pop_sec_total(const PopArgs& a) { return min(*a.sec_count, a.sec_cap); }
__device__ __forceinline__ bool claimed(const unsigned int* claim, int i) { return (claim[i >> 5] >> (i & 31)) & 1u; }

// Each phase is a list of items per slot (its length from the slot's counts
// as the previous phases left them). The grid works through all slots' items
// in 32-item warp chunks, so a warp's lanes always belong to one slot (the
// warp-aggregated appends and growth sums stay within it).
struct PopPlan {
  int pre[kBatchMaxSlots + 1];  // exclusive prefix of the slots' chunk counts
  int items[kBatchMaxSlots];
  int warp[kPopThreads / 32];
};

// exclusive block-wide prefix sum of v (every thread calls it); *total = the sum
__device__ __forceinline__ int block_exclusive_sum(int v, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int w = lane < nw ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) s_warp[lane] = w;
  }
  __syncthreads();
  const int off = wid ? s_warp[wid - 1] : 0;
  *total = s_warp[nw - 1];
  __syncthreads();
  return off + x - v;
}

// the phase's item counts and chunk prefix in shared memory; returns the chunks
template <class Src, class Items>
__device__ __forceinline__ int pop_plan(const Src& src, int n, Items items, PopPlan& pl) {
  int carry = 0;
  for (int base = 0; base < n; base += blockDim.x) {
    const int s = base + threadIdx.x;
    int k = 0;
    if (s < n) {
      const PopArgs* ap = src.get(s);
      k = ap ? max(items(*ap), 0) : 0;
      pl.items[s] = k;
    }
    int tot = 0;
    const int ex = block_exclusive_sum((k + 31) >> 5, pl.warp, &tot);
    if (s < n) pl.pre[s] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) pl.pre[n] = carry;
  __syncthreads();
  return carry;
}

// body(a, i) for every item i of every slot
template <class Src, class Items, class Body>
__device__ __forceinline__ void pop_phase(const Src& src, PopPlan& pl, Items items, Body body) {
  const int n = src.count();
  const int total = pop_plan(src, n, items, pl);
  const int lane = threadIdx.x & 31;
  const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), GW = (int)((gridDim.x * blockDim.x) >> 5);
  for (int c = gw; c < total; c += GW) {
    int lo = 0, hi = n;  // largest s with pre[s] <= c
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (pl.pre[mid] <= c) lo = mid;
      else hi = mid;
    }
    const int i = ((c - pl.pre[lo]) << 5) + lane;
    if (i < pl.items[lo]) body(*src.get(lo), i);
  }
}

__device__ __forceinline__ int pop_attached(const PopArgs& a) { return *a.att_count; }
// attached slots and left-over secondaries (items of the first phase), and how many
// more there are of one than of the other (items of the others)
__device__ __forceinline__ int pop_left(const PopArgs& a) { return abs(pop_attached(a) - pop_sec_total(a)); }

// items of the first phase: the attached slots and the removal draws
__device__ __forceinline__ int pop_fill_items(const PopArgs& a) { return max(pop_attached(a), pop_sec_total(a)); }

__device__ __forceinline__ void pop_fill_item(const PopArgs& a, int i) {
  const int n_att = pop_attached(a), n_sec = pop_sec_total(a);
  if (i < n_att) {
    const int slot = a.att_list[i];
    if (i < n_sec) {
      const int k = n_sec - 1 - i;
      a.state[2 * slot] = a.sec[2 * k];
      a.state[2 * slot + 1] = a.sec[2 * k + 1];
    } else {
      atomicOr(&a.claim[slot >> 5], 1u << (slot & 31));
    }
    return;
  }
  const int j = i - n_att, pool = a.n_electrons + (n_sec - n_att);
  const uint64_t interval = a.ctl->interval;
  int got = -1;
  for (uint32_t d = 0; d < 4096u; ++d) {
    const int r = uniform_index(pop_word((uint32_t)j, interval, a.seed, 2u, d), pool);
    const unsigned int bit = 1u << (r & 31);
    const unsigned int old = atomicOr(&a.claim[r >> 5], bit);
    if (!(old & bit)) {
      got = r;
      break;
    }
  }
  a.removed[j] = got;
  if (got < 0) atomicExch(a.error_flag, 5);
}

// the drain's shared memory: the process constants stay in global memory
using DrainShared = AdvSharedT<kPopThreads / 32, 32, 1>;

template <class Src>
__global__ void __launch_bounds__(kPopThreads) k_pop_fill(const __grid_constant__ Src src) {
  __shared__ DrainShared sh;
  __shared__ AdvanceArgs s_a;
  __shared__ PopPlan pl;
  next_may_start();
  wait_for_previous();
  // (a slot's spill count is final here except for its own drain, which only raises it)
  auto spilled = [](const AdvanceArgs& a) { return *(volatile const int*)a.spill_count != 0; };
  for (int s = blockIdx.x; s < src.count(); s += gridDim.x) {
    const PopArgs* a = src.get(s);
    if (!a || !spilled(*src.advance(s))) continue;
    __syncthreads();
    load_slot_args(src.advance(s), &s_a);
    __syncthreads();
    drain_body(s_a, sh);
    for (int i = threadIdx.x; i < pop_fill_items(*a); i += blockDim.x) pop_fill_item(*a, i);
  }
  pop_phase(
      src, pl,
      [&](const PopArgs& a) { return *(volatile const int*)a.spill_count != 0 ? 0 : pop_fill_items(a); },
      [](const PopArgs& a, int i) { pop_fill_item(a, i); });
}

template <class Src>
__global__ void __launch_bounds__(kPopThreads) k_pop_clone(Src src) {
  __shared__ PopPlan pl;
  next_may_start();
  wait_for_previous();
  pop_phase(src, pl, pop_left, [](const PopArgs& a, int item) {
    const int n_att = pop_attached(a), n_sec = pop_sec_total(a);
    if (n_att > n_sec) {
      const int j = n_sec + item;
      const int dest = a.att_list[j];
      const uint64_t interval = a.ctl->interval;
      int src_slot = -1;
      for (uint32_t d = 0; d < 4096u; ++d) {
        const int r = uniform_index(pop_word((uint32_t)j, interval, a.seed, 1u, d), a.n_electrons);
        if (!claimed(a.claim, r) && a.state[2 * r + 1].w == 0.0f) {
          src_slot = r;
          break;
        }
      }
      if (src_slot < 0) {
        atomicExch(a.error_flag, 4);
        return;
      }
      const float4 A = a.state[2 * src_slot], B = a.state[2 * src_slot + 1];
      a.state[2 * dest] = A;
      a.state[2 * dest + 1] = B;
      add_growth(a.growth, (double)energy4(B, a.half_me_over_e));
      return;
    }
    const int r = a.removed[item];
    if (r >= 0 && r < a.n_electrons) {
      a.pair_slot[append_slot(&a.counts[0])] = r;
      add_growth(a.growth, -(double)energy4(a.state[2 * r + 1], a.half_me_over_e));
    } else if (r >= a.n_electrons) {
      add_growth(a.growth, -(double)energy4(a.sec[2 * (r - a.n_electrons) + 1], a.half_me_over_e));
    }
    if (!claimed(a.claim, a.n_electrons + item)) a.pair_sec[append_slot(&a.counts[1])] = item;
  });
}

template <class Src>
__global__ void __launch_bounds__(kPopThreads) k_pop_place(Src src) {
  __shared__ PopPlan pl;
  next_may_start();
  wait_for_previous();
  pop_phase(src, pl, pop_left, [](const PopArgs& a, int item) {
    const int n_att = pop_attached(a), n_sec = pop_sec_total(a);
    if (n_att > n_sec) {
      const int dest = a.att_list[n_sec + item];
      atomicAnd(&a.claim[dest >> 5], ~(1u << (dest & 31)));
      return;
    }
    // as many secondaries survive as slots were removed, unless a draw gave up
    if (item < min(a.counts[0], a.counts[1])) {
      const int slot = a.pair_slot[item], k = a.pair_sec[item];
      a.state[2 * slot] = a.sec[2 * k];
      a.state[2 * slot + 1] = a.sec[2 * k + 1];
    }
    const int r = a.removed[item];
    if (r >= 0) atomicAnd(&a.claim[r >> 5], ~(1u << (r & 31)));
  });
}

template <class Src>
void launch_pop_phases(const Src& src, int grid, bool after_kernel, cudaStream_t s) {
  launch_after(k_pop_fill<Src>, grid, kPopThreads, 0, s, after_kernel, src);
  launch_after(k_pop_clone<Src>, grid, kPopThreads, 0, s, true, src);
  launch_after(k_pop_place<Src>, grid, kPopThreads, 0, s, true, src);
}

// ---------------------------------------------------------- batch helpers
// distribution tallies of the slots that sample them this interval
// the chunk this block takes in round r (snake order, lgpu_chunks.h)
__device__ __forceinline__ int snake_chunk(int r) { return snake_index(r, gridDim.x, blockIdx.x); }

__global__ void __launch_bounds__(kHistAThreads) k_hist_a_batch(BatchArgs b) {
  extern __shared__ unsigned int sm_hist[];
  const int n_slots = b.hdr->n_slots, total = b.hdr->hist_chunks, n_full = b.hdr->hist_full;
  for (int r = 0; r * (int)gridDim.x < total; ++r) {
    const int c = snake_chunk(r);
    if (c >= total) continue;
    const ChunkRef k = pass_chunk(b.hist_prefix, b.hist_part, n_slots, n_full, b.hdr->hist_chunk, c);
    const HistArgs& a = b.hists[k.slot];
    hist_chunk_a(a, k.first, min(k.first + b.hdr->hist_chunk, a.n), sm_hist, kHistASmem / 4);
  }
}

__global__ void __launch_bounds__(kHistBThreads) k_hist_b_batch(BatchArgs b) {
  extern __shared__ unsigned int sm_hist[];
  const int n_slots = b.hdr->n_slots, total = b.hdr->hist2_chunks, n_full = b.hdr->hist2_full;
  for (int r = 0; r * (int)gridDim.x < total; ++r) {
    const int c = snake_chunk(r);
    if (c >= total) continue;
    const ChunkRef k = pass_chunk(b.hist2_prefix, b.hist2_part, n_slots, n_full, b.hdr->hist_chunk, c);
    const HistArgs& a = b.hists[k.slot];
    hist_chunk_b(a, k.first, min(k.first + b.hdr->hist_chunk, a.n), sm_hist, kHistBSmem / 4);
  }
}

// Moments of the sampling slots and, in the same read, the distributions of the
// slots whose sample records them on a grid that holds (DistCtl), in chunks of
// hdr->smp_chunk electrons.
//
// The 64-point sweep: moments with the EVDF, then EEDF and EADF in a pass of their
// own, took 123 + 195 us per interval; all of it takes 177 here (3.6 TB/s), of which the
// addition of every chunk's occupied cells to the tallies at L2 35, the shared additions
// 10 to 30 and the read alone 93; the launch waits for the blocks with two whole chunks
// (1.17 of the mean share). 32 conditions of 10,000-30,000
// electrons: 21 + 66 -> 25 us. Loads in flight are not what it waits for: a ring of
// asynchronous copies in place of the four records in registers took 193.
constexpr int kSampleBatchShared = 8192;  // electrons of a chunk that are worth shared cells (16 jobs: 41 us, 56 with 16384)

__global__ void __launch_bounds__(kSampleSharedThreads) k_sample_batch(BatchArgs b) {
  __shared__ double s_m[kSampleSharedThreads / 32][kMoments];
  extern __shared__ unsigned int sm_dist[];
  next_may_start();
  wait_for_previous();
  const int n_slots = b.hdr->n_slots, total = b.hdr->smp_chunks, n_full = b.hdr->smp_full, chunk = b.hdr->smp_chunk;
  for (int r = 0; r * (int)gridDim.x < total; ++r) {
    const int c = snake_chunk(r);
    if (c >= total) continue;
    const ChunkRef k = pass_chunk(b.smp_prefix, b.smp_part, n_slots, n_full, chunk, c);
    const BatchSlot& sl = b.slots[k.slot];
    if (!sl.ctl.go) continue;  // its chain has stopped
    const SampleArgs& a = sl.smp;
    const int last = min(k.first + chunk, a.n);
    if (sl.dist.on && __uint_as_float(sl.sc->max_energy_bits) <= sl.dist.e_bound) {
      const bool shared = last - k.first >= kSampleBatchShared;
      sample_counting(a, sl.dist.h, shared, k.first + threadIdx.x, last, blockDim.x, s_m, sm_dist);
    } else {
      sample_range(a, k.first + threadIdx.x, last, blockDim.x, s_m);
    }
    __syncthreads();
  }
}

// the end of the interval: one block per slot, and the advance's time
constexpr int kBatchEndThreads = 128;

__global__ void __launch_bounds__(kBatchEndThreads) k_batch_end(BatchArgs b) {
  next_may_start();
  wait_for_previous();
  BatchHeader& h = *b.hdr;
  const int s = blockIdx.x;
  if (s == 0 && threadIdx.x == 0) {
    if (h.advance_end) {  // a slot ran
      b.out->advance_ns[h.pos] = (double)(h.advance_end - h.advance_begin);
      b.out->intervals = h.pos + 1;
    }
    ++h.pos;
    h.advance_begin = ~0ull;
    h.advance_end = 0ull;
  }
  BatchSlot& sl = b.slots[s];
  end_interval(ThisBlock(), sl.ctl, sl.dist, sl.chain, sl.sc, sl.adv.n, b.gather + s, b.max_slots, &b.out->done[s],
               &b.out->stopped, (sl.flags & kSlotSample) != 0);
}

// --------------------------------------------------------------- replay
__global__ void k_replay_flight(ReplayFlightArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  float3 p = make_float3((float)a.pos[3 * i], (float)a.pos[3 * i + 1], (float)a.pos[3 * i + 2]);
  float3 v = make_float3((float)a.vel[3 * i], (float)a.vel[3 * i + 1], (float)a.vel[3 * i + 2]);
  const float e0 = energy_of(v, a.half_me_over_e);
  free_flight(a.field, (float)a.phi0[i], (float)a.dt[i], p, v);
  const float e1 = energy_of(v, a.half_me_over_e);
  a.pos_out[3 * i] = p.x;
  a.pos_out[3 * i + 1] = p.y;
  a.pos_out[3 * i + 2] = p.z;
  a.vel_out[3 * i] = v.x;
  a.vel_out[3 * i + 1] = v.y;
  a.vel_out[3 * i + 2] = v.z;
  a.energy_out[i] = e1;
  a.gain_out[i] = e1 - e0;
}

__global__ void k_replay_collide(ReplayCollArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  ReplayStream rng;
  rng.u = a.u + (size_t)i * a.u_stride;
  rng.n = a.u_stride;
  rng.pos = 0;
  float3 v = make_float3((float)a.vel[3 * i], (float)a.vel[3 * i + 1], (float)a.vel[3 * i + 2]);
  float energy = (float)a.energy[i];
  CollResult cr;
  cr.ej_v = make_float3(0.f, 0.f, 0.f);
  if (a.coarse) {
    // the advance kernels' event: the null test tries the block bound of the
    // total frequency first (lane_flight), then the rest of the collision
    // (lane_real)
    float r = 0.0f;
    const float nu = (float)a.nu[i];
    if (is_thermal(a.c, energy) || cold_real(a.t, nu, energy, rng, r, a.t.nu_coarse)) {
      collide_pending(a.c, a.t, a.procs, a.gases, nu, r, v, energy, rng, cr);
    } else {
      cr.chosen = -1;
      cr.dE = 0.0f;
      cr.ionized = 0;
    }
  } else {
    collide(a.c, a.t, a.procs, a.gases, (float)a.nu[i], v, energy, rng, cr);
  }
  double* o = a.out + (size_t)i * 11;
  o[0] = cr.chosen;
  o[1] = v.x;
  o[2] = v.y;
  o[3] = v.z;
  o[4] = energy;
  o[5] = cr.chosen >= 0 ? cr.dE : 0.0;
  o[6] = cr.chosen >= 0 ? (double)cr.dE / a.energy[i] : 0.0;
  const bool ion = cr.chosen >= 0 && cr.ionized;
  o[7] = ion ? cr.ej_v.x : 0.0;
  o[8] = ion ? cr.ej_v.y : 0.0;
  o[9] = ion ? cr.ej_v.z : 0.0;
  o[10] = ion ? (double)energy_of(cr.ej_v, a.c.half_me_over_e) : 0.0;
  a.used[i] = rng.pos;
}

template <int BLOCKS_PER_SM>
void launch_advance_modes(const AdvanceArgs& args, bool after_kernel, cudaStream_t s) {
  AdvanceArgs a = args;
  // blocks of two warps while that puts at most four warps on an SM: 24 -> 22.5 us at 10,000
  const int threads = a.n <= a.sm_count * 4 * 32 ? 64 : kAdvanceThreads;
  const int warps = threads / 32, per_sm = BLOCKS_PER_SM * kAdvanceThreads / threads;
  const int grid = max(1, min(a.sm_count * per_sm, (a.n + threads - 1) / threads));
  const int all = grid * warps;
  a.share = a.n <= all * 32 ? 32 : (int)(0.8 * a.n / all) / 32 * 32;
  switch (a.field.mode) {
    case kFieldDC: launch_after(k_advance<kFieldDC, BLOCKS_PER_SM>, grid, threads, 0, s, after_kernel, a); break;
    case kFieldAC: launch_after(k_advance<kFieldAC, BLOCKS_PER_SM>, grid, threads, 0, s, after_kernel, a); break;
    case kFieldB: launch_after(k_advance<kFieldB, BLOCKS_PER_SM>, grid, threads, 0, s, after_kernel, a); break;
    case kFieldECR: launch_after(k_advance<kFieldECR, BLOCKS_PER_SM>, grid, threads, 0, s, after_kernel, a); break;
    default: launch_after(k_advance<kFieldACB, BLOCKS_PER_SM>, grid, threads, 0, s, after_kernel, a); break;
  }
}

inline int blocks_for(int n, int threads) { return (n + threads - 1) / threads; }

}  // namespace

// The main pass over one condition's ensemble. The electrons are spread over all
// warps the device holds: one per lane while they last (an electron's events follow
// one another, so a second electron of the lane only adds to the longest chain),
// else each warp starts on four fifths of an even share and takes the rest 32 at a
// time. Every warp taking 128 at a time from a counter instead kept one SM in 15
// busy with 10,000 electrons, and left the last chunks to a few warps at 1e6:
// 10,000 electrons (atomic gas, DC) 38 -> 23 us, 33,333 (Reid) 34 -> 17, 100,000
// (mixture, crossed B, thermal) 58 -> 38, 1e6 (N2-like) 85 -> 74, 4e6 unchanged
// at 194. The collision stash of the batched shapes waits for 32 collisions at the
// end of every condition and is no faster here (79 us at 1e6, 194 at 4e6).
//
// While one electron per lane needs fewer lanes than four blocks per SM hold, two or
// three blocks hold them all, with the registers of the others: no spills, and more
// of an electron's chain of loads and divisions side by side. 10,000 electrons (atomic
// gas) 15.4 -> 14.5 us, 33,333 (Reid) 10.8 -> 10.0 by the device's clock with two;
// 100,000 (mixture, crossed B, thermal) 31.7 -> 30.3 with three.
void launch_advance(const AdvanceArgs& a, bool after_kernel, cudaStream_t s) {
  const int lanes = a.sm_count * kAdvanceThreads;  // of one block per SM
  if (a.n <= 2 * lanes) launch_advance_modes<2>(a, after_kernel, s);
  else if (a.n <= 3 * lanes) launch_advance_modes<3>(a, after_kernel, s);
  else launch_advance_modes<kAdvanceBlocksPerSM>(a, after_kernel, s);
}

void launch_init(const InitArgs& a, cudaStream_t s) {
  if (a.n <= 0) return;
  k_init<<<blocks_for(a.n, 256), 256, 0, s>>>(a);
}

// A block that has its SM to itself, because there are no more blocks than SMs or because
// two blocks' values do not fit one, takes 32 warps instead of 8: its processes'
// interpolations are chains of dependent loads and divisions. Whole calls with 8 and 32:
// 100 rows of 196 processes 121 and 84 us, of 410 215 and 150; 1000 rows 174 and 138, 327 and
// 268; 4864 rows of 40 and 410 105 and 103, 835 and 769, 10,000 of 410 1765 and 1619. With
// several blocks to an SM the small ones leave it sooner: 10,000 rows of 40 processes 182
// and 193, of 65 285 and 300.
void launch_build_tables(const TableBuildArgs& a, int sm_count, cudaStream_t s) {
  const int blocks = blocks_for(a.M, kTableRows), smem = table_smem(a.P);
  if (blocks <= sm_count || 2 * smem > 227 * 1024) k_build_tables<kTableThreadsAlone><<<blocks, kTableThreadsAlone, smem, s>>>(a);
  else k_build_tables<kTableThreads><<<blocks, kTableThreads, smem, s>>>(a);
  const int bounds = a.nu_coarse ? blocks_for(a.n_coarse, kPrefixThreads / 32) : 0;
  k_table_bounds<<<1 + bounds, kPrefixThreads, 0, s>>>(a.nu_tot, a.nu_max, a.M, a.nu_pair, a.coarse_shift, a.nu_coarse,
                                                       a.n_coarse);
}

// Blocks of the single-condition sample: half-size ones while the ensemble does
// not fill the device with full ones (they clear and add up their EEDF counts
// side by side; 10,000 electrons with distributions 9.1 -> 7.1 us), full ones
// from there (fewer EEDF additions per electron: 200,000 electrons under AC
// 21.9 -> 15.9 us), one large one per SM with EADF and EVDF cells in shared memory
// from kSampleShared electrons per SM on, 798,000 on 152 SMs. Below, clearing and
// adding up the shared cells costs more than the additions at L2 that they save: per
// interval with and without them, atomic gas DC 62.4 and 59.2 us at 450,000, 68.6 and 65.7
// at 600,000, 77.8 and 77.1 at 800,000, 86.3 and 86.7 at 1e6; N2-like 77.1 and 75.9, 85.2
// and 83.9, 94.1 and 95.4, 103.4 and 107.3.
constexpr int kSampleShared = 5250;

void launch_sample(const SampleArgs& a, int sm_count, bool after_kernel, cudaStream_t s) {
  if (a.n <= 0) return;
  const int sms = max(1, sm_count);
  const bool shared = a.plain && a.n >= sms * kSampleShared && a.n <= sms * 64512ll;  // below 2^16 a block
  if (shared) {
    launch_after(k_sample<true>, min(blocks_for(a.n, kSampleSharedThreads), sms), kSampleSharedThreads, kSampleSmem, s,
                 after_kernel, a);
    return;
  }
  const int threads = a.n < sms * kSampleThreads ? kSampleThreads / 2 : kSampleThreads;
  const int grid = min(blocks_for(a.n, threads), sms * (1024 / threads));
  launch_after(k_sample<false>, grid, threads, a.plain ? a.dist_e_cells * sizeof(unsigned int) : 0, s, after_kernel,
               a);
}

void launch_rebin(const RebinArgs& a, cudaStream_t s) {
  k_rebin<<<1 + a.n_cos + a.n_phases, kRebinThreads, a.n_e * kRebinCell, s>>>(a);
}

void launch_interval_end(const SampleArgs& a, cudaStream_t s) { launch_after(k_interval_end, 1, 128, 0, s, true, a); }

void launch_hist(const HistArgs& a, cudaStream_t s) {
  if (a.n <= 0) return;
  const int chunks = (a.n + kHistChunk - 1) / kHistChunk;
  k_hist_a<<<chunks, kHistAThreads, kHistASmem, s>>>(a);
  if (a.cylindrical) k_hist_b<<<chunks, kHistBThreads, kHistBSmem, s>>>(a);
}

void launch_pop_control(const AdvanceArgs& adv, const PopArgs& a, cudaStream_t s) {
  PopOne one;
  one.a = a;
  one.adv = adv;
  launch_pop_phases(one, kPopBlocks, true, s);
}

cudaError_t prepare_kernels() {
  static_assert(table_smem(kMaxProcesses) <= 227 * 1024, "the tables of the most processes fit a block");
  cudaError_t e = cudaFuncSetAttribute(k_build_tables<kTableThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, table_smem(kMaxProcesses));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_build_tables<kTableThreadsAlone>, cudaFuncAttributeMaxDynamicSharedMemorySize, table_smem(kMaxProcesses));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_a, cudaFuncAttributeMaxDynamicSharedMemorySize, kHistASmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_hist_b, cudaFuncAttributeMaxDynamicSharedMemorySize, kHistBSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_hist_a_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, kHistASmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_hist_b_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, kHistBSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sample_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleSmem);
  static_assert(kMaxEnergyCells * kRebinCell <= 227 * 1024, "the cells of a column fit a block");
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rebin, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxEnergyCells * kRebinCell);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sample<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleSmem);
  if (e == cudaSuccess) e = prepare_advance_stash();
  return e;
}

size_t batch_prefix_offset() { return (sizeof(BatchHeader) + 15) / 16 * 16; }
size_t batch_slots_offset() {
  return (batch_prefix_offset() + (4 * (kBatchMaxSlots + 1) + 3 * kBatchMaxSlots) * sizeof(int) + 255) / 256 * 256;
}

int launch_batch_hist(const BatchArgs& b, int sm_count, unsigned parts, cudaStream_t s) {
  int n = 0;
  if (parts & kPartHistA) {
    k_hist_a_batch<<<sm_count, kHistAThreads, kHistASmem, s>>>(b);
    ++n;
  }
  if (parts & kPartHistB) {
    k_hist_b_batch<<<sm_count * 2, kHistBThreads, kHistBSmem, s>>>(b);
    ++n;
  }
  return n;
}

int launch_batch_post(const BatchArgs& b, int sm_count, int n_slots, unsigned parts, bool after_kernel,
                      cudaStream_t s) {
  int n = 1;
  if (parts & kPartIonAtt) {
    PopBatch pb;
    pb.hdr = b.hdr;
    pb.slots = b.slots;
    launch_pop_phases(pb, sm_count * kPopBlocksPerSM, after_kernel, s);
    n += kPopLaunches;
    after_kernel = true;
  }
  if (parts & kPartSample) {
    launch_after(k_sample_batch, sm_count, kSampleSharedThreads, kSampleSmem, s, after_kernel, b);
    ++n;
    after_kernel = true;
  }
  launch_after(k_batch_end, n_slots, kBatchEndThreads, 0, s, after_kernel, b);
  return n;
}

void launch_replay_flight(const ReplayFlightArgs& a, cudaStream_t s) {
  if (a.n > 0) k_replay_flight<<<blocks_for(a.n, 128), 128, 0, s>>>(a);
}

void launch_replay_collide(const ReplayCollArgs& a, cudaStream_t s) {
  if (a.n > 0) k_replay_collide<<<blocks_for(a.n, 128), 128, 0, s>>>(a);
}

}  // namespace lgpu
