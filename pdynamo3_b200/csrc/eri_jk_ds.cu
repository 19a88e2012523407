// Coulomb/exchange kernels with a (ds| bra.
#include "eri_jk.cuh"

PDG_JK_ROW(3, launch_jk_t<3, 0>, launch_jk_t<3, 1>, launch_jk_t<3, 2>, launch_jk_t<3, 3>)
