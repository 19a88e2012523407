// Coulomb/exchange kernels with a (dd| bra.
#include "eri_jk.cuh"

PDG_JK_ROW(5, launch_jk_t<5, 0>, launch_jk_t<5, 1>, launch_jk_t<5, 2>, launch_jk_t<5, 3>, launch_jk_t<5, 4>, launch_jk_t<5, 5>)
