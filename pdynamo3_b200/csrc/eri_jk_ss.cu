// Coulomb/exchange kernels with a (ss| bra.
#include "eri_jk.cuh"

PDG_JK_ROW(0, launch_jk_t<0, 0>)
