// Coulomb/exchange kernels with a (ps| bra.
#include "eri_jk.cuh"

PDG_JK_ROW(1, launch_jk_t<1, 0>, launch_jk_t<1, 1>)
