/* count32_box.cu -- instantiations of the FP32 counting kernel for one
 * periodic box (one catalogue pair per launch). */
#include "tile32.cuh"

kfun_t fcfcg_pick32_box(int bin, int wt) {
#define K32(B)                                                             \
  if (bin == B)                                                            \
    return wt ? (kfun_t) k_tile32<FCFCG_GEOM_BOX, B, 1, 0>       \
              : (kfun_t) k_tile32<FCFCG_GEOM_BOX, B, 0, 0>;
  K32(FCFCG_BIN_ISO)
  K32(FCFCG_BIN_SMU)
  K32(FCFCG_BIN_SPI)
  K32(BIN_SPILIN)
  K32(BIN_ISOLIN)
  K32(BIN_SMULIN)
#undef K32
  return 0;
}
