// Host-side helpers shared by the translation units of libgbgpu_gb300.
#pragma once

#include <cuda_runtime.h>

int set_error(int code, const char *fmt, ...);
int cuda_error(cudaError_t e, const char *what);
int num_sms();
int ensure_init(cudaStream_t st);
int gbx_twiddle_init(cudaStream_t st);

// Prepares `kern` for launches of `block` threads with `smem` bytes of dynamic
// shared memory on the current device and gives what fits: the resident blocks per
// SM or, for clusters of `cluster` blocks, the resident clusters (0: it cannot be
// launched so, as on a partition of a GPU).
int kernel_fit(const void *kern, int block, size_t smem, int *fit, int cluster = 1);

// A launch in clusters; `attr` has to live as long as the configuration is used.
cudaLaunchConfig_t cluster_config(unsigned grid, int cluster, int block, size_t smem, cudaLaunchAttribute *attr);
