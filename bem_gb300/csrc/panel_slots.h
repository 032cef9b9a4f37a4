// Where the warps of a panel CTA keep their candidates of a column (dense.cu,
// panel_cluster_kernel).  A column has one barrier, between the candidates' writes
// and their reads; what follows it waits only for the message of the warp that
// owns the CTA's candidate.  A warp may therefore write its candidate of the next column
// while another still reads this column's: the next column uses another set.  Two
// sets do: whoever writes column j + 2 has passed the barrier of column j + 1, and
// so has every reader of column j.
#pragma once

#ifdef __CUDACC__
#define PANEL_SLOTS_HD __host__ __device__
#else
#define PANEL_SLOTS_HD
#endif

constexpr int PANEL_SLOT_SETS = 2;
PANEL_SLOTS_HD constexpr int panel_slot_set(int column) { return column % PANEL_SLOT_SETS; }
