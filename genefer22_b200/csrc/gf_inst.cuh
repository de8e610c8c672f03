// gf_inst.cuh -- the kernel templates' instances, in groups.
//
// Each group is compiled in a source file of its own (gf_inst_*.cu, explicit
// instantiations) and declared extern in gf_host.cu, which launches them: the
// files compile in parallel (one file took eight minutes).
#pragma once

#include "gf_kernels.cuh"

#define GFC_SMALL_N(T, SET, LOGN) T void k_small<SET, LOGN, false>(const Args);
#define GFC_SMALL_S(T, SET, LOGN) T void k_small<SET, LOGN, true>(const Args);
#define GFC_INST_SMALL(T)                                                                                              \
	GFC_SMALL_N(T, ANY_SET, 10) GFC_SMALL_S(T, ANY_SET, 10) GFC_SMALL_N(T, ANY_SET, 11) GFC_SMALL_S(T, ANY_SET, 11)    \
	GFC_SMALL_N(T, 0, 12) GFC_SMALL_S(T, 0, 12) GFC_SMALL_N(T, 1, 12) GFC_SMALL_S(T, 1, 12)                            \
	GFC_SMALL_N(T, 3, 12) GFC_SMALL_S(T, 3, 12) GFC_SMALL_N(T, ANY_SET, 12) GFC_SMALL_S(T, ANY_SET, 12)                \
	GFC_SMALL_N(T, 0, 13) GFC_SMALL_N(T, 1, 13) GFC_SMALL_N(T, 3, 13) GFC_SMALL_N(T, ANY_SET, 13)                      \
	GFC_SMALL_N(T, 0, 14) GFC_SMALL_N(T, 1, 14) GFC_SMALL_N(T, 3, 14) GFC_SMALL_N(T, ANY_SET, 14)

#define GFC_CLUSTER(T, LQ, LC, SET) T void k_cluster<LQ, LC, SET>(const Args, int);
#define GFC_INST_CLUSTER_SHORT(T)                                                                                      \
	GFC_CLUSTER(T, 3, 9, 0) GFC_CLUSTER(T, 3, 9, 3) GFC_CLUSTER(T, 3, 9, ANY_SET)                                      \
	GFC_CLUSTER(T, 4, 9, 0) GFC_CLUSTER(T, 4, 9, 3) GFC_CLUSTER(T, 4, 9, ANY_SET)                                      \
	GFC_CLUSTER(T, 4, 10, 0) GFC_CLUSTER(T, 4, 10, 3) GFC_CLUSTER(T, 4, 10, ANY_SET)
#define GFC_INST_CLUSTER_LONG(T)                                                                                       \
	GFC_CLUSTER(T, 2, 13, 0) GFC_CLUSTER(T, 2, 13, ANY_SET)                                                            \
	GFC_CLUSTER(T, 3, 13, 0) GFC_CLUSTER(T, 3, 13, ANY_SET) GFC_CLUSTER(T, 4, 13, 0) GFC_CLUSTER(T, 4, 13, ANY_SET)

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
