// Internal hooks between the host engine (fr_capi.cu), the serving layer (fr_server.cu) and
// the autotuner (fr_tune.cu).
#pragma once

#include "umpalumpa_fr.h"

namespace frb {

// Sticky device-side status (FR_OK or an FR_E_* code) as copied back by the handle's last
// finished batched launch; valid once that launch's work has completed on the stream.
int batch_device_status(const fr_handle *h);

// Initialises the handle again for the same strategy, from `held` in place of the caller's launch
// parameters (nullptr: from those), so that the item buffer and grid follow.
int reinit(fr_handle *h, const fr_launch_params *held);

// Autotuner hooks (fr_tune.cu).  tune_lookup: the launch parameters the handle's last search found
// for its current strategy (dims/limits and settings set), else, unless the approach is
// FR_TUNING_OFF, those of the strategy's tuning file, if it exists.  tune_single:
// the search of fr_autotune, run by fr_execute under FR_TUNING_ON_EXECUTE.
bool tune_lookup(const fr_handle *h, fr_launch_params *out);
int tune_single(fr_handle *h, const void *fft, const float *scales, uint64_t nProj,
  const fr_traverse_space *spaces, uint64_t nSpaces, const float *table, fr_tune_report *report);

}// namespace frb
