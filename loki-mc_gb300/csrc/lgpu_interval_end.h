// lgpu_interval_end.h - the end of one interval of a chain, by the threads of one
// block: usable from device code and, with threads of the host in their place, from
// host C++ alike.
#pragma once

#include <cstddef>

#include "lgpu_kernels.cuh"

namespace lgpu {

LGPU_HD float float_of_bits(unsigned int bits) {
  union {
    unsigned int u;
    float f;
  } x;
  x.u = bits;
  return x.f;
}

// The end of an interval of one condition with n electrons (every thread of one block
// calls this; all other work of the interval is done), unless its chain has stopped
// before: its scalars go to the host (out[pos * stride]), the ones of one interval are
// cleared, and the next interval of the chain is set up or the chain stopped (then
// *stopped, where given, is 1).
//
// Block: thread() of threads(), sync() as a barrier for all of them, load(p) for what
// other blocks have written. Every thread reads `go` and the position, which thread 0
// goes on to change, ahead of the first barrier.
template <class Block>
LGPU_HD void end_interval(const Block& b, IntervalCtl& ctl, DistCtl& dist, ChainCtl& ch, DevScalars* sc, int n,
                          DevScalars* out, int stride, int* done, int* stopped, bool sampled) {
  const int go = ctl.go, pos = ch.pos;
  b.sync();
  if (!go) return;
  constexpr int kWords = (int)(sizeof(DevScalars) / sizeof(int));
  const int* src = reinterpret_cast<const int*>(sc);
  int* dst = reinterpret_cast<int*>(&out[(size_t)pos * stride]);
  for (int k = b.thread(); k < kWords; k += b.threads()) dst[k] = b.load(&src[k]);
  if (b.thread() == 0) {
    const float e = float_of_bits(b.load(&sc->sample_max_bits));
    const bool counted = !dist.on || float_of_bits(b.load(&sc->max_energy_bits)) <= dist.e_bound;
    const bool more = sampled && pos + 1 < ch.n && counted && e >= ch.e_lo && e <= ch.e_hi &&
                      b.load(&sc->error_flag) == 0 && b.load(&sc->sec_count) <= ch.sec_stop;
    if (more) {
      // the host's arithmetic: the FP64 mean, rounded to FP32
      ctl.shift_x = (float)(b.load(&sc->moments[1]) / (double)n);
      ctl.shift_y = (float)(b.load(&sc->moments[2]) / (double)n);
      ctl.shift_z = (float)(b.load(&sc->moments[3]) / (double)n);
      ctl.phi0 = ch.phi0[pos + 1];
      ++ctl.interval;
      dist.h.eedf_periodic_row = ch.row[pos + 1];
      ch.pos = pos + 1;
    } else {
      ctl.go = 0;
      if (stopped) *stopped = 1;
    }
    *done = pos + 1;
  }
  b.sync();
  for (int k = b.thread(); k < (int)(offsetof(DevScalars, null_count) / sizeof(int)); k += b.threads())
    reinterpret_cast<int*>(sc)[k] = 0;
  for (int k = b.thread(); k < kMoments; k += b.threads()) sc->moments[k] = 0.0;
  if (b.thread() == 0) sc->sample_max_bits = 0u;
}

}  // namespace lgpu
