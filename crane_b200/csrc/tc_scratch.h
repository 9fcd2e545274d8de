// Per-stream scratch of the tensor-core kernels: partial tiles, arrival counters (zero between launches) and the bounded waits' error word.
// Kernels on one stream are ordered (and a programmatic dependent only touches the scratch after its dependency wait), so one set per stream
// is enough.  Host code only.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

namespace cb {

constexpr size_t TC_WS_FLOATS = (size_t)2 * 160 * 128 * 256;     // two partial 128 x 256 tiles per CTA

struct TcScratch { float* ws = nullptr; int* counters = nullptr; int* err = nullptr; };

// Scratch of `st` with at least `n_counters` counters.  What was handed out stays where it is until tc_scratch_release: captured graphs hold the
// addresses.  So a call for more counters gets a second, larger block beside the first (powers of two: all blocks together are under twice the
// largest).  May be called while `st` is being captured in relaxed mode.  0, or a CUDA error.
int tc_scratch_get(cudaStream_t st, int n_counters, TcScratch* out);
// the error word alone (kernels that share no tiles)
int tc_err_word(cudaStream_t st, int** out);
// true once if a wait of a kernel on `st` ran out since the last call (read after a synchronisation of the stream)
bool tc_take_wait_error(cudaStream_t st);
// Frees the scratch kept for `st`: after its last kernel and its graphs, before the stream is destroyed.
void tc_scratch_release(cudaStream_t st);

}  // namespace cb
