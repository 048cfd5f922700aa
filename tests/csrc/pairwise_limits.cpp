/* The limits of gba_pairwise_6d behind a C face. */
#include "../../gpuattract_2.0_gb300/csrc/pairwise_limits.h"

extern "C" int pairwise_refuses(int backward, uint32_t num_types, uint32_t n_lig, uint32_t n_rec) {
	return gba::pairwise_refused(backward != 0, num_types, n_lig, n_rec) != nullptr;
}
