/* count32_f64.cu -- instantiations of the tile kernel with every pair in FP64
 * (counts and adjoint). */
#include "tile32.cuh"

kfun_t fcfcg_pick64(int geom, int wt, int adj) {
#define K64(G)                                                             \
  (adj ? (kfun_t) k_tile32<G, BIN_F64, 1, 0, 1>                            \
       : (wt ? (kfun_t) k_tile32<G, BIN_F64, 1, 0>                         \
             : (kfun_t) k_tile32<G, BIN_F64, 0, 0>))
  return geom == FCFCG_GEOM_BOX ? K64(FCFCG_GEOM_BOX) : K64(FCFCG_GEOM_SURVEY);
#undef K64
}
