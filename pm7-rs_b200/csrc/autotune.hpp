// Autotuner of result-identical launch variants (autotune.cpp).
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <string>

namespace pm7 {

// Launches variant launch(v) of `key` on stream st. On the first use of `key` on this device
// (and with no entry in the PM7_AUTOTUNE_CACHE file) every variant is run once untimed and
// once timed with CUDA events, synchronously, and the fastest is kept; afterwards only the
// kept variant is launched; PM7_AUTOTUNE_FORCE="prefix=variant,..." overrides both for keys
// with that prefix. Returns the variant used. Every variant must write the same results. Not
// for use inside a stream capture.
int autotune(cudaStream_t st, const std::string &key, int n_variants, const std::function<void(int)> &launch);

// The same for launches that can be refused (cooperative ones): launch(v) returns its status, which
// this returns too. While timing, a variant whose launch fails is passed over and never kept; when all
// fail nothing is kept and the first status is returned. alike: the variants of this key are one and
// the same launch, so there is nothing to time: variant 0 is kept.
cudaError_t autotune_checked(cudaStream_t st, const std::string &key, int n_variants,
                             const std::function<cudaError_t(int)> &launch, int *used = nullptr, bool alike = false);

// The decisions so far as JSON ({"<device>|<key>": variant, ...}).
std::string autotune_report();

}  // namespace pm7
