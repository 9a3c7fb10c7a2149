// lgpu_kernels.cuh - launch interface of the electron Monte Carlo kernels
// (implemented in lgpu_kernels.cu, called by the host runtime).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "lgpu_chunks.h"
#include "lgpu_types.h"

namespace lgpu {

constexpr int kMaxProcesses = 512;
constexpr int kMaxGases = 16;
constexpr int kMaxEnergyCells = 4096;
constexpr int kMoments = 22;  // sum e, r(3), v(3), r r^T (6 unique), r v^T (9)

// Device scalars of one condition, read back after every interval.
// Per-interval fields first (cleared before every interval), cumulative after.
struct DevScalars {
  int sec_count, att_count, spill_count, error_flag;
  unsigned int max_energy_bits;
  int work_counter;
  int pop_counts[2];    // population control: removed slots, surviving secondaries
  // device clock (ns) at which block 0 of the advance starts and its last block ends
  // (one condition per launch)
  unsigned long long advance_begin, advance_end;
  unsigned long long null_count;
  unsigned long long real_count;
  double field_gain;
  double growth;
  double time_adjust;   // electron-time beyond N x interval: + secondaries, - attachments (s)
  unsigned int sample_max_bits;
  int pad2;
  double moments[kMoments];
};

// Arguments of one advance launch: every electron of the ensemble is pushed
// from the start of the synchronisation interval to its end, colliding on the
// way; secondaries created on the way are queued and pushed from their
// creation time to the end of the interval by the same launch.
struct AdvanceArgs {
  float4* state;            // [2*N]: (x, y, z, s) and (vx, vy, vz, dead flag) per electron
  int n;                    // electrons of the ensemble
  float dt_sync;            // interval length (s)
  float phi0;               // phase at the interval start (rad), FP64-reduced on the host
  float phase_rate;         // w (AC, AC+B) or W (resonance)
  float nu;                 // trial collision frequency (1/s)
  uint64_t seed;
  uint64_t interval;        // synchronisation interval index (random-number counter)
  uint32_t salt;
  float3 shift;             // origin shift subtracted from every position on load
  FieldF field;
  Consts c;
  TablesF t;
  const ProcF* procs;
  const GasF* gases;
  int P;
  // secondaries pushed to the end of the interval: (x, y, z, s), (vx, vy, vz, 0)
  float4* sec;
  int* sec_count;
  int sec_cap;
  // secondaries a warp could not keep in its own queue: (x, y, z, t_c), (vx, vy, vz, 0)
  float4* spill;
  int* spill_count;
  int spill_cap;
  int* att_list;                   // attached ensemble slots
  int* att_count;
  unsigned long long* proc_count;  // [P]
  double* proc_gain;               // [P]
  double* proc_loss;               // [P]
  unsigned long long* null_count;
  unsigned long long* real_count;
  double* field_gain;
  double* time_adjust;             // simulated electron-time beyond N * dt: + secondaries, - attachments (s)
  unsigned int* max_energy_bits;   // float bits of the largest final energy
  int* error_flag;                 // 2: secondary buffer full, 3: collision budget exhausted
  int* work_counter;               // chunk counter of the persistent grid (zero before the launch)
  int sm_count;
  const IntervalCtl* ctl;          // when set: per-interval values are read from here
  int real_batch;                  // pending real collisions that start a warp's collision turn (1..32)
  int coarse;                      // 1: null test against the block bounds first (t.nu_coarse)
  int local_q;                     // secondaries a warp queues before it spills (1..kLocalQ)
  // one condition per launch: the electrons each warp starts on (set by
  // launch_advance) and the device clock of the launch
  int share;
  unsigned long long *advance_begin, *advance_end;
};
// Lanes with a pending collision that start a warp's collision turn. Cold gases take
// their null test in the flight, so that the lanes that wait idle through other
// lanes' flights: 16 (4e6 electrons, atomic gas: 168 us, 176 with 20, 190 with 24; 1e6,
// N2-like: 62 at 16 and 20, 65 at 24). With thermal targets every event waits for the
// turn: 20 (1e6, mixture under crossed B: 95 us, 99 with 16, 94 with 24).
constexpr int kRealBatchCold = 16, kRealBatchThermal = 20;

// after_kernel: as launch_after's
void launch_advance(const AdvanceArgs& a, bool after_kernel, cudaStream_t s);

// Per-process kernel attributes (dynamic shared memory of the histogram
// kernels); called on the current device before any launch or capture.
cudaError_t prepare_kernels();

struct InitArgs {
  float4* state;
  int n;
  float sd;                 // sqrt(k T_e / m)
  uint64_t seed;
  float half_me_over_e;
  unsigned int* max_energy_bits;
};
void launch_init(const InitArgs& a, cudaStream_t s);

// Table build on the device in FP64 (BoltzmannMC.C:561-615).
struct TableBuildArgs {
  int M, P, stride;
  double step, N;
  const int* is_super;
  const double* superw;
  const double* emin;
  const double* emax;
  const double* rel_dens;
  const int* raw_off;
  const int* raw_len;
  const double* raw_e;
  const double* raw_v;
  float2* nu_pair;
  float2* cum_pair;
  float2* sig_pair;
  double* nu_tot;     // FP64 total frequency per row
  double* nu_max;     // FP64 running maximum
  double* sig64;      // optional FP64 sigma*n [M*P] (tests), may be null
  double* cum64;      // optional FP64 cumulative [M*P] (tests), may be null
  float* nu_coarse;   // block bounds for the coarse null test [n_coarse], may be null
  int coarse_shift, n_coarse;
};
void launch_build_tables(const TableBuildArgs& a, int sm_count, cudaStream_t s);

// Distribution tallies of one sample (BoltzmannMC.C:1550-1571).
struct HistArgs {
  const float4* state;
  int n;
  float half_me_over_e;
  int n_e_cells;
  float inv_e_step;                // 1 / EEDF energy step
  double* eedf;                    // [n_e_cells]
  double* eedf_periodic_row;       // [n_e_cells] or null
  int cylindrical;
  int n_cos;                       // EADF: [n_e_cells x n_cos]
  double* eadf;
  int n_rad, n_ax;                 // EVDF: [n_rad x n_ax]
  float inv_rad_step, inv_ax_step, max_speed;
  double* evdf;
};
// The tallies on the energy grid moved to a wider one (BoltzmannMC.C:1495-1548).
struct RebinArgs {
  int n_e, n_cos, n_phases;        // n_cos 0: no EADF; n_phases 0: no per-phase EEDFs
  double old_step, old_max, step;  // the grids' cell widths, the old one's maximum
  double* eedf;                    // [n_e]
  double* eadf;                    // [n_e x n_cos]
  double* eedf_per;                // [n_phases x n_e]
};
void launch_rebin(const RebinArgs& a, cudaStream_t s);

// What the sample of an interval counts beside its moments, written by the host
// with the interval's control block: the distributions (BoltzmannMC.C:1550-1571)
// when their energy grid holds every electron. Whether it does is known before
// the sample: no electron at the end of the interval is above the largest energy
// the advance saw (population control only drops and copies electrons), so the
// sample counts when that energy is at most `e_bound`, the largest float on the
// grid, and otherwise leaves the tallies to the host, which re-bins first.
struct DistCtl {
  int on;
  float e_bound;
  HistArgs h;
};

// Ensembles of a context on its own up to this size count their distributions with
// the sample: above it a block of one per SM would see more electrons than its 16-bit
// counts hold, and the passes over 65535-electron chunks fill the device. The passes come
// before the next interval's advance, so that such intervals are chains of their own.
constexpr int kDistInSample = 9000000;

// A chain of intervals of one condition: the host launches up to kChain of them
// without a look in between. At the end of each the device keeps the interval's
// scalars for the host, clears them and writes the next interval's control block
// (the origin shift is the new ensemble mean), or stops the chain, whose launches
// left then do nothing for the condition, when the host has something to do first: a
// look at the trial frequency or energy tables (the largest energy left [e_lo,
// e_hi]), a re-binning, larger buffers, or an error to report.
constexpr int kChain = 16;

struct ChainCtl {
  int n;                      // intervals of the chain
  int pos;                    // index of the one being run
  float e_lo, e_hi;
  int sec_stop;               // more secondaries than this stop the chain
  float phi0[kChain];         // the intervals' phases
  double* row[kChain];        // their samples' per-phase EEDF rows
};

// what the host sends before a chain of a context on its own
struct PlainCtl {
  IntervalCtl ctl;            // the interval being run
  DistCtl dist;
  ChainCtl chain;
  unsigned int ticket;        // blocks of the sample that are done (left zero)
};

// where a chain's scalars go: host memory the device can write
struct ChainOut {
  int done;                   // intervals run
  int pad[3];
  DevScalars sc[kChain];
};

// Ensemble sample: moment sums (FP64) and the largest energy, and, with `plain`,
// the distributions in the same read of the ensemble and the end of the interval.
struct SampleArgs {
  const float4* state;
  int n;
  float half_me_over_e;
  double* moments;                 // [kMoments], accumulated (zero on entry)
  unsigned int* max_energy_bits;
  PlainCtl* plain;                 // null: moments only
  DevScalars* sc;                  // the condition's scalars (with plain)
  ChainOut* out;
  int dist_e_cells;                // EEDF cells (with plain)
};
// the end of an interval without a sample, behind its other kernels
void launch_interval_end(const SampleArgs& a, cudaStream_t s);
// grid: at most four blocks per SM (sm_count = the device's multiprocessors)
void launch_sample(const SampleArgs& a, int sm_count, bool after_kernel, cudaStream_t s);

void launch_hist(const HistArgs& a, cudaStream_t s);

// Population control (BoltzmannMC.C:1282-1408) at the end of an interval,
// when every electron and every secondary is at the synchronisation time.
struct PopArgs {
  float4* state;
  int n_electrons;
  const float4* sec;               // advanced secondaries (x, y, z, s), (vx, vy, vz, dead flag)
  const int* sec_count;            // may exceed sec_cap after an overflow (reported by the host)
  const int* spill_count;          // secondaries that the warps could not queue
  int sec_cap;
  int* counts;                     // [2] zero on entry: removed slots, surviving secondaries
  const int* att_list;
  const int* att_count;
  unsigned int* claim;             // bitmap over n_electrons + sec_cap, all zero on entry and on exit
  int* removed;                    // [sec_cap] scratch
  int* pair_slot;                  // [sec_cap] scratch
  int* pair_sec;                   // [sec_cap] scratch
  double* growth;                  // energy growth accumulator (eV)
  float half_me_over_e;
  uint64_t seed;
  const IntervalCtl* ctl;
  int* error_flag;                 // set when a bounded retry loop gives up
};
// The secondaries the warps could not queue (adv: the advance's arguments), then
// three launches (filling of attached slots and removal draws, clones or listing,
// pairing), each spread over many blocks.
void launch_pop_control(const AdvanceArgs& adv, const PopArgs& a, cudaStream_t s);
constexpr int kPopLaunches = 3;

// ------------------------------------------------------------------ batches
// Many swarm conditions (slots) advanced by one launch sequence per interval.
// Each slot carries the same argument blocks a single-condition launch takes;
// the kernels split every slot's ensemble into fixed-size chunks and find the
// slot of a chunk by bisection over exclusive prefix sums of the chunk counts.
enum SlotFlags : int { kSlotIonAtt = 1, kSlotSample = 2 };

struct BatchSlot {
  AdvanceArgs adv;        // adv.ctl points at this slot's ctl (the device's copy)
  PopArgs pop;
  SampleArgs smp;
  DistCtl dist;           // distributions counted with this interval's sample
  IntervalCtl ctl;        // this interval's values
  ChainCtl chain;
  DevScalars* sc;         // the condition's scalars; the per-interval part is zero before an interval
  int flags;              // SlotFlags
  int pad;
};

constexpr int kFieldModes = 5;

// Slots are ordered by field mode; the advance runs one launch per mode over
// that mode's slots [mode_slot[m], mode_slot[m + 1]).
struct BatchHeader {
  int n_slots;
  int adv_chunks, smp_chunks, hist_chunks;  // totals (last prefix entries)
  int mode_chunk[kFieldModes + 1];          // first advance chunk of each mode's slots
  int mode_slot[kFieldModes + 1];           // first slot of each mode
  int hist2_chunks;                         // velocity-distribution chunks (cylindrical slots)
  // the moment and distribution passes list each slot's full chunks first
  // (prefix over slots) and then one partial chunk per slot, largest first,
  // so that the blocks' static shares of the list come out even
  int smp_full, hist_full, hist2_full;
  int smp_chunk, hist_chunk;                // electrons per chunk of the samples and of the histograms
  int pos;                                  // index of the interval in the chain
  // device clock (ns) at which the first branch's block 0 starts the advance and the last
  // block of any ends it
  unsigned long long advance_begin, advance_end;
};

// Where a chain of batched intervals goes: host memory the device can write. The
// advance publishes the index of the interval it begins: what the intervals before it
// wrote can then be read, while it runs.
constexpr int kBatchChain = kChain;
struct BatchOut {
  int published;                            // -1 before the chain
  int stopped;                              // a slot's chain has stopped
  int intervals;                            // launched intervals in which a slot ran
  int pad;
  double advance_ns[kBatchChain];
  int done[1024];                           // intervals each slot ran (kBatchMaxSlots)
};

constexpr int kBatchMaxSlots = 1024;
constexpr int kBatchAdvanceChunk = 4096;   // granularity of the advance's initial spread of blocks over slots
constexpr int kBatchSampleChunk = 65535;   // electrons per chunk of the samples at most (16-bit EVDF counts)
constexpr int kBatchHistChunk = 65535;     // electrons per chunk of the histograms at most (16-bit counts)
// Batches of fewer sampled electrons count their distributions in passes of their own, an
// interval at a time, as all batches did once. It is not what is faster for them: one
// pass and chains take a served job of 50,000 electrons from 40 to 20 ms. The check that
// arriving jobs overlap on the device (tests/test_gpu_batch.py) has them arrive 38 ms apart.
constexpr double kBatchDistMin = 150000;

// Staging layout (host pinned mirror and device copy are identical):
//   BatchHeader | adv_prefix | smp_prefix | hist_prefix | hist2_prefix (kBatchMaxSlots+1 ints
//   each) | smp_part | hist_part | hist2_part (kBatchMaxSlots ints each, padded) | BatchSlot[...]
// The interval's staging fills the advance and moment parts, the distribution
// passes' staging the hist parts and, in place of the slots, the deferred tallies of a
// previous sample (HistArgs[...]).
struct BatchArgs {
  BatchHeader* hdr;
  BatchSlot* slots;
  const HistArgs* hists;    // (distribution passes)
  const int* adv_prefix;
  const int* smp_prefix;    // full chunks before each slot
  const int* hist_prefix;   // energy and energy-angle distributions
  const int* hist2_prefix;  // velocity distribution (cylindrical slots)
  const int* smp_part;      // slots with a partial chunk, largest partial first
  const int* hist_part;
  const int* hist2_part;
  DevScalars* gather;       // [kBatchChain x max_slots]: each slot's scalars after each interval
  BatchOut* out;
  int max_slots;
};
size_t batch_prefix_offset();   // bytes from the staging start to adv_prefix
size_t batch_slots_offset();    // bytes from the staging start to slots[0]
static_assert(kBatchMaxSlots == 1024 && kBatchChain <= kChain, "BatchOut, ChainCtl");
// One batched interval is two launch groups on one stream:
//   advance: one persistent launch per field mode
//   post:    spilled secondaries and population control, samples, the interval's end
// ahead of a chain of them, from a second staging area, the distribution passes of the
// previous interval's samples, launched before the host prepares the interval so that its work
// runs beside them.
// `parts` leaves out the launches no slot of the interval needs: bit m (m <
// kFieldModes) for field mode m, then the flags below. Each returns the
// kernels it launched.
enum BatchParts : unsigned {
  kPartHistA = 1u << 8,   // a slot records its energy distributions
  kPartHistB = 1u << 9,   // a slot records its velocity distribution in a separate pass
  kPartSample = 1u << 10, // a slot samples its moments
  kPartIonAtt = 1u << 11, // a slot has ionization or attachment (spilled secondaries, population control)
};
int launch_batch_hist(const BatchArgs& b, int sm_count, unsigned parts, cudaStream_t s);
// The batched advance in one of kAdvShapes launch shapes (threads per block,
// blocks per SM, electrons a warp takes at a time, records of a warp's
// collision stash); advance_shape() names them. Shapes from 4 on are stash
// shapes (lgpu_advance_stash.cu).
constexpr int kAdvShapes = 6;
constexpr int kFirstStashShape = 4;
int launch_batch_advance(const BatchArgs& b, int sm_count, unsigned parts, int shape, bool after_kernel,
                         cudaStream_t s);
int launch_batch_advance_stash(const BatchArgs& b, int sm_count, unsigned parts, int shape, bool after_kernel,
                         cudaStream_t s);
void advance_shape(int shape, int* threads, int* blocks_per_sm, int* chunk, int* stash);
// dynamic shared memory of the stash shapes' kernels (part of prepare_kernels)
cudaError_t prepare_advance_stash();
// after_kernel: the last work on the stream is a kernel of this interval
int launch_batch_post(const BatchArgs& b, int sm_count, int n_slots, unsigned parts, bool after_kernel, cudaStream_t s);

// End-of-job EEDF post-processing in FP64 (lgpu_post.cu): the EEDF-convolved
// rate coefficient of every MC process (Collision.C:355-397) for each of
// n_eedf EEDFs, and, unless rates_only, the two-term swarm parameters
// (BoltzmannMC.C:2186-2266) of the one EEDF given.
struct EedfPostArgs {
  int nc, P, n_eedf, rates_only;
  double max_energy, gas_density, omega, omega_c;
  const double* eedf_in;   // normalised EEDFs [n_eedf][nc], or null: normalise eeh
  const double* eeh;       // histogram sums [n_eedf][nc]
  const int* kind;         // per process: 0 elastic, 1 inelastic, 2 superelastic copy
  const int* ion;          // 1 ionization, 2 attachment
  const double* dens;      // target (product) relative density
  const double* thr;       // threshold (eV)
  const double* mass_ratio;
  const double* stat;      // g_target / g_product
  const int* int_off;
  const int* int_len;
  const int* mom_off;
  const int* mom_len;
  const double* raw_ie;
  const double* raw_iv;
  const double* raw_me;
  const double* raw_mv;
  double* eedf_norm;       // [n_eedf][nc]: the normalised EEDFs when eeh is given
  double* shares;          // [3][P][nc + 1]: each process's share of the node totals (unless rates_only)
  double* sums;            // [eedf_post_sums(nc)]: block sums of the parameters (unless rates_only)
  double* parts;           // [P][n_eedf][tiles]: the rates' sums over tiles of cells
  unsigned int* ticket;    // [1 + P] zero before the first call, left zero by each
  double* rates;           // [n_eedf][P]
  double* out;             // host memory: the rates, then [16] parameters (lgpu_eedf_params order)
};
size_t eedf_post_sums(int nc);
int eedf_post_tile(int nc, int P, int sm_count);  // cells of a tile
// returns the kernels it launched
int launch_eedf_post(const EedfPostArgs& a, int sm_count, cudaStream_t s);

// Replay kernels for the parity tests: the production device functions
// driven by given inputs and recorded uniforms.
struct ReplayFlightArgs {
  int n;
  const double* phi0;     // phase at flight start (rad, already reduced)
  const double* dt;
  const double* pos;      // [n*3]
  const double* vel;      // [n*3]
  double* pos_out;
  double* vel_out;
  double* energy_out;
  double* gain_out;
  FieldF field;
  float half_me_over_e;
};
void launch_replay_flight(const ReplayFlightArgs& a, cudaStream_t s);

struct ReplayCollArgs {
  int n;
  const double* nu;
  const double* vel;      // [n*3]
  const double* energy;
  const double* u;        // [n*u_stride]
  int u_stride;
  double* out;            // [n*11]: chosen, v(3), energy, dE, dE/E, ej v(3), ej energy
  int* used;
  Consts c;
  TablesF t;
  const ProcF* procs;
  const GasF* gases;
  int coarse;             // 1: the null test of the advance kernels (block bounds first)
};
void launch_replay_collide(const ReplayCollArgs& a, cudaStream_t s);

}  // namespace lgpu
