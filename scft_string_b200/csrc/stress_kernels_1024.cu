// stress_kernels_1024.cu -- the kernels of stress_kernels.cu for CTAs of up to 1024 threads.
#define SCFT_STRESS_THREADS 1024
#include "stress_kernels.cu"
