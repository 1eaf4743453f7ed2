// stress_kernels_512.cu -- the kernels of stress_kernels.cu for CTAs of up to 512 threads.
#define SCFT_STRESS_THREADS 512
#include "stress_kernels.cu"
