// gf_inst.cuh -- the kernel templates' instances, in groups.
//
// Each group is compiled in a source file of its own (gf_inst_*.cu, explicit
// instantiations) and declared extern in gf_host.cu, which launches them: the
// files compile in parallel (one file took eight minutes).
#pragma once

#include "gf_kernels.cuh"

#define GFC_SMALL_N(T, SETS, LOGN) T void k_small<SETS, LOGN, false>(const Args);
#define GFC_SMALL_S(T, SETS, LOGN) T void k_small<SETS, LOGN, true>(const Args);
#define GFC_SMALL_SETS(G, T, LOGN)                                                                                     \
	G(T, SETS_0, LOGN) G(T, SETS_1, LOGN) G(T, SETS_01, LOGN) G(T, SETS_3, LOGN) G(T, SETS_03, LOGN) G(T, SETS_ANY, LOGN)
#define GFC_INST_SMALL(T)                                                                                              \
	GFC_SMALL_SETS(GFC_SMALL_N, T, 10) GFC_SMALL_SETS(GFC_SMALL_S, T, 10) GFC_SMALL_SETS(GFC_SMALL_N, T, 11)           \
	GFC_SMALL_SETS(GFC_SMALL_S, T, 11) GFC_SMALL_SETS(GFC_SMALL_N, T, 12) GFC_SMALL_SETS(GFC_SMALL_S, T, 12)           \
	GFC_SMALL_SETS(GFC_SMALL_N, T, 13) GFC_SMALL_SETS(GFC_SMALL_N, T, 14)

#define GFC_CLUSTER(T, LQ, LC, SETS) T void k_cluster<LQ, LC, SETS>(const Args, int);
#define GFC_CLUSTER_S(T, LQ, LC)                                                                                       \
	GFC_CLUSTER(T, LQ, LC, SETS_01) GFC_CLUSTER(T, LQ, LC, SETS_3) GFC_CLUSTER(T, LQ, LC, SETS_03)                     \
	GFC_CLUSTER(T, LQ, LC, SETS_ANY)
#define GFC_INST_CLUSTER_SHORT(T) GFC_CLUSTER_S(T, 3, 9) GFC_CLUSTER_S(T, 4, 9) GFC_CLUSTER_S(T, 4, 10)
#define GFC_INST_CLUSTER_LONG(T)                                                                                       \
	GFC_CLUSTER(T, 2, 13, SETS_01) GFC_CLUSTER(T, 2, 13, SETS_ANY) GFC_CLUSTER(T, 3, 13, SETS_01)                      \
	GFC_CLUSTER(T, 3, 13, SETS_ANY) GFC_CLUSTER(T, 4, 13, SETS_01) GFC_CLUSTER(T, 4, 13, SETS_ANY)

#define GFC_COL(T, LR) T void k_col_fwd<LR>(const Args); T void k_col_inv<LR>(const Args);
#define GFC_INST_COL(T) GFC_COL(T, 5) GFC_COL(T, 6) GFC_COL(T, 7) GFC_COL(T, 8) GFC_COL(T, 9) GFC_COL(T, 10)

#define GFC_COLR(T, LR, S3)                                                                                            \
	T void k_colr_fwd<LR, S3>(const Args); T void k_colr_inv<LR, S3>(const Args);                                      \
	T void k_colr_fwd_s<LR, S3>(const Args); T void k_colr_inv_s<LR, S3>(const Args);
#define GFC_INST_COLR(T) GFC_COLR(T, 3, false) GFC_COLR(T, 3, true) GFC_COLR(T, 4, false) GFC_COLR(T, 4, true)

#define GFC_ROW(T, LC) T void k_row<LC, false>(const Args); T void k_row<LC, true>(const Args);
#define GFC_ROW_PAIR(T, LC) T void k_row2<LC>(const Args, int); T void k_rowp<LC>(const Args);
#define GFC_INST_ROW(T) GFC_ROW(T, 8) GFC_ROW(T, 9) GFC_ROW(T, 10) GFC_ROW(T, 11) GFC_ROW(T, 12) GFC_ROW(T, 13)
#define GFC_INST_ROW_PAIR(T)                                                                                           \
	GFC_ROW_PAIR(T, 8) GFC_ROW_PAIR(T, 9) GFC_ROW_PAIR(T, 10) GFC_ROW_PAIR(T, 11) GFC_ROW_PAIR(T, 12) GFC_ROW_PAIR(T, 13)

#define GFC_MIDR(T, LR2, S3) T void k_midr<LR2, false, S3>(const Args); T void k_midr<LR2, true, S3>(const Args);
#define GFC_INST_MID(T)                                                                                                \
	GFC_MIDR(T, 3, false) GFC_MIDR(T, 3, true) GFC_MIDR(T, 4, false) GFC_MIDR(T, 4, true) GFC_MIDR(T, 5, false)        \
	GFC_MIDR(T, 5, true) T void k_midp<false, false>(const Args); T void k_midp<false, true>(const Args);              \
	T void k_midp<true, false>(const Args); T void k_midp<true, true>(const Args); T void k_mid<7, false>(const Args); \
	T void k_mid<7, true>(const Args);

#define GFC_PCOL(T, LR)                                                                                                \
	T void k_pcol_fwd<LR>(const Args); T void k_pcol_inv<LR>(const Args);                                              \
	T void k_pcol_fwd_s<LR, PCS_MINB_HI>(const Args); T void k_pcol_inv_s<LR, PCS_MINB_HI>(const Args);                \
	T void k_pcol_fwd_s<LR, PCS_MINB_LO>(const Args); T void k_pcol_inv_s<LR, PCS_MINB_LO>(const Args);
#define GFC_INST_PCOL(T) GFC_PCOL(T, 3) GFC_PCOL(T, 4)
