// Explicit (ab|c) block kernels of the bra class L_ab = 2 (every auxiliary L).
#include "k_std3c_impl.cuh"

PA_STD3C_ROW(2)
