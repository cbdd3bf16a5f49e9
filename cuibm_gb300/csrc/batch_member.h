// What the batch (batch.cpp) needs of an instance beyond the C ABI: its step recorded into
// the batch's step graph, and the host side of the steps the batch graph ran (context.cu).
#pragma once
#include <cuda_runtime.h>

#include "../../include/cuibm.h"

extern "C" {
// Which of the instance's step graphs is current (each has a number of its own), or 0 when its
// steps need host work between them (no step graph, per-phase profiling, or a hierarchy
// rebuilt as an embedded body moves).
unsigned long long cuibm_batch_member_graph(cuibm_ctx *h);
// Record the instance's step into the capture under way on stream `on`, as a branch of its own
// between `fork`, recorded there, and the stream's next work.
int cuibm_batch_member_record(cuibm_ctx *h, cudaStream_t on, cudaEvent_t fork);
// The instance's stream (its work outside the batch graph runs there).
cudaStream_t cuibm_batch_member_stream(cuibm_ctx *h);
// Account for n steps the batch graph ran for the instance.
void cuibm_batch_member_advance(cuibm_ctx *h, int n);
}
