// Device-side state that the launchers of the attention kernels share: the split-KV workspace and
// arrival counters of a stream, the self-resetting scheduler words, the SM count.  Defined in
// paged_attention.cu.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "../../include/b200pa.h"

namespace b200pa {

constexpr int kArrivePerRegion = 32768;

struct StreamRegion {
  unsigned char* ws;   // split-KV workspace of this stream
  size_t ws_bytes;
  unsigned* arrive;    // arrival counters of this stream (kArrivePerRegion, zero between launches)
  unsigned* arrive2;   // ... of its merge groups
};

bool stream_region(cudaStream_t stream, StreamRegion* out);
unsigned* sched_words(cudaStream_t stream);
int sm_count();

// paged_attention_v1 on the first half of the stream's workspace and arrival counters; the attention
// entries directly behind the KV write of their step (see launch_dependent).
int attention_half_region(const b200pa_attn_args* a, void* stream, bool behind_write);
int attention_behind_write(const b200pa_attn_args* a, void* stream, bool caller_scratch);
// Whether paged_attention_v1 (v2 with `caller_scratch`) takes the call, without launching anything.
int attention_check(const b200pa_attn_args* a, bool caller_scratch);

}  // namespace b200pa
