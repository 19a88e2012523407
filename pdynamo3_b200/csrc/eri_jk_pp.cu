// Coulomb/exchange kernels with a (pp| bra.
#include "eri_jk.cuh"

PDG_JK_ROW(2, launch_jk_t<2, 0>, launch_jk_t<2, 1>, launch_jk_t<2, 2>)
