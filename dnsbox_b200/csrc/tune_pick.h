// The autotuner's last decision (host code; no CUDA).
#pragma once

// The fastest of the n uniform schedules by their measured step times and of the
// schedule composed of each pass's fastest kernel: the index of the uniform run,
// or -1 for the composed one.  A pass's time depends on the others' kernels (the
// compact workspace rows need all four strided passes on the SIMT kernel), so a
// composed schedule may be slower than the runs its passes come from.
inline int fastest_schedule(const double *uniform_ms, int n, double composed_ms) {
  int best = -1;
  double ms = composed_ms;
  for (int i = 0; i < n; ++i)
    if (uniform_ms[i] < ms) ms = uniform_ms[i], best = i;
  return best;
}
