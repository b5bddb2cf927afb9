// Launch of the drain kernel (drain.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

struct DevCtx;
struct SchedState;

constexpr int kDrainThreads = 128;

// Blocks of the drain kernel resident per SM; head: the plan has jaws or an MLC.
int drain_blocks_per_sm(bool head);
void launch_drain(const DevCtx &C, SchedState *st, bool head, int grid, cudaStream_t s);
