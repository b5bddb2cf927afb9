// Launch of the drain kernel (drain.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

struct DevCtx;
struct SchedState;

constexpr int kDrainThreads = 128;

// Blocks of the drain kernel resident per SM; head: the plan has jaws or an MLC.
int drain_blocks_per_sm(bool head);
// Memory for the frames of all threads that the device can hold of it, with what
// else a launch may need.
size_t drain_frames(bool head);
void launch_drain(const DevCtx &C, SchedState *st, bool head, int grid, cudaStream_t s);
