// mesh-solve kernels of order 5
#include "ct2g_fft_mesh.cuh"

CT2G_FFT_ORDER_FNS(5)
