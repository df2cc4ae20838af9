// batch_kernel20.cu -- the batched engine's persistent kernel for ranks 2..20.
#include "batch_run.cuh"

#include "batch_kernel.cuh"

nmfb_batched::BatchKernel nmfb_batched::batch_kernel20() { return k_batch<20>; }
