// batch_kernel10.cu -- the batched engine's persistent kernel for ranks 2..10.
#include "batch_run.cuh"

#include "batch_kernel.cuh"

nmfb_batched::BatchKernel nmfb_batched::batch_kernel10() { return k_batch<10>; }
