/*
 * mhd_layout.h -- slots of the FP32 forms' state arrays (U, V, the fluxes, ...).
 *
 * A row of cells along z takes kp slots, a multiple of MHD_GROUP, with k = 1 on
 * a group's first slot; k = 0 takes the last, otherwise unused, slot of the row
 * before (MHD_GROUP slots lead the first row).  The nine variables of a group
 * lie together, [slot / MHD_GROUP][m][slot % MHD_GROUP], so a cell's variables
 * are one address and eight constant offsets, where [m][cells] costs a 64-bit
 * address for every variable and neighbour, and neighbours along r and phi are
 * whole groups away.
 *
 * Groups of 8 are the smallest that are whole 32-byte sectors: a warp's 32
 * cells are four of them, none shared with another row's.  Rounding a row up to
 * groups of 32, one aligned 128-byte line, costs up to 31 slots a row in every
 * array (kz = 32: 64 slots for 34 cells, with 8: 40) and reads the sectors
 * between a row's end and its neighbour's ghost.  A step in FP32, groups of 32
 * / 16 / 8: 256x256x12 802 / 688 / 683 us, 256x256x32 878 / 860 / 831,
 * 256x256x48 1381 / 1324 / 1296, 256x256x128 2624 / 2613 / 2615, 151x90x77 (MC)
 * 497 / 469 / 469, 64x64x32 109 / 106 / 105; 512x512x256 19.08 / 19.00 / 19.35
 * ms (pair state 24.32 / 24.29 / 24.59), where the rounding is small and four
 * lines a load cost more than they save.  The same bits throughout.
 *
 * Plain C++: the host compiles it too, for the tests.
 */
#ifndef MHD_LAYOUT_H
#define MHD_LAYOUT_H

#ifdef __CUDACC__
#define MHD_LAYOUT_FN __host__ __device__ __forceinline__
#else
#define MHD_LAYOUT_FN static inline
#endif

/* slots whose nine variables lie together, and slots per tile of the update
 * staged by bulk copies (a multiple of it) */
#define MHD_GROUP 8
#define MHD_UPD_TILE 128

namespace mhd {

/* slots of a row of kzmax cells */
MHD_LAYOUT_FN int row_slots(int kzmax) { return (kzmax + MHD_GROUP - 1) / MHD_GROUP * MHD_GROUP; }
/* slots of an array of `rows` rows */
MHD_LAYOUT_FN long long array_slots(long long rows, int kp) { return MHD_GROUP + rows * kp; }
/* the slot of cell k of a row, and the offset of a slot's first variable */
MHD_LAYOUT_FN long long row_slot(long long row, int kp, int k) { return row * kp + (k + MHD_GROUP - 1); }
MHD_LAYOUT_FN long long slot_offset(long long q) { return q + 8 * (q & ~(long long)(MHD_GROUP - 1)); }

} /* namespace mhd */

#endif
