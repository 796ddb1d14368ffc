/* count32_adj.cu -- instantiations of the FP32 tile kernel's adjoint
 * (gradients of weighted counts with respect to the weights). */
#include "tile32.cuh"

kfun_t fcfcg_pick32_adj(int geom, int bin) {
#define K32A(G, B)                                                         \
  if (geom == G && bin == B) return (kfun_t) k_tile32<G, B, 1, 0, 1>;
#define K32G(G)                                                            \
  K32A(G, FCFCG_BIN_ISO)                                                   \
  K32A(G, FCFCG_BIN_SMU)                                                   \
  K32A(G, FCFCG_BIN_SPI)                                                   \
  K32A(G, BIN_SPILIN)                                                      \
  K32A(G, BIN_ISOLIN)                                                      \
  K32A(G, BIN_SMULIN)
  K32G(FCFCG_GEOM_BOX)
  K32G(FCFCG_GEOM_SURVEY)
#undef K32G
#undef K32A
  return 0;
}
