/*
 * pairwise_limits.h -- what a gba_pairwise_6d call may ask for, decided on the
 * host before anything is launched.  Plain C++, in 64 bits: the kernels count
 * a block's cells in 32 bits, which the sizes accepted here never leave.
 */
#ifndef GBA_PAIRWISE_LIMITS_H_
#define GBA_PAIRWISE_LIMITS_H_

#include <cstddef>
#include <cstdint>

namespace gba {

/* Bead types have 16 bits (gba_upload_protein), and a table's T * T entries
 * are numbered in 32. */
constexpr uint32_t kPairwiseMaxTypes = 65535;

/* The backward pass's cells of one block at most. */
constexpr size_t kPairwiseCellBytes = 200 * 1024 - 8 * 2624;

/* Bytes of a block's cells: two per type pair, one per ligand and receptor
 * bead.  num_types <= kPairwiseMaxTypes. */
inline size_t pairwise_cell_bytes(uint32_t num_types, uint32_t n_lig, uint32_t n_rec) {
	return (2 * (size_t)num_types * num_types + n_lig + n_rec) * sizeof(uint64_t);
}

/* Why a call is refused, or nullptr. */
inline const char* pairwise_refused(bool backward, uint32_t num_types, uint32_t n_lig, uint32_t n_rec) {
	if (num_types > kPairwiseMaxTypes) return "gba_pairwise_6d: num_types > 65535";
	if (backward && pairwise_cell_bytes(num_types, n_lig, n_rec) > kPairwiseCellBytes)
		return "gba_pairwise_6d: proteins/types too large for the adjoint's shared partials";
	return nullptr;
}

}  // namespace gba

#endif /* GBA_PAIRWISE_LIMITS_H_ */
