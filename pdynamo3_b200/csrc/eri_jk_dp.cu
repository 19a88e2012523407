// Coulomb/exchange kernels with a (dp| bra.
#include "eri_jk.cuh"

PDG_JK_ROW(4, launch_jk_t<4, 0>, launch_jk_t<4, 1>, launch_jk_t<4, 2>, launch_jk_t<4, 3>, launch_jk_t<4, 4>)
