// stage_variants.h -- launch shapes of the fused stage kernel per N.
// Each entry X(KS, EPB, KSMEM, MINB, ALG): KS threads per node column, EPB
// elements per block, KSMEM = stage k in shared memory (1) or read it from L2
// after a prefetch (0), MINB = resident blocks the register allocator must
// allow, ALG = 0 for the SIMT tile (stage_kernel.cuh), 1 for the FP64
// tensor-core tile (stage_mma.cuh: N = 8, FP64 only), 201 for the field-split FP64 tensor-core tile (stage_dmma.cuh: N = 8,
// axis-aligned class, FP64 only), or 2 + flags for the second family (stage_pipe.cuh; KSMEM must be 0) with flags
// 1 = PIPE (persistent, double-buffered), 2 = SPLIT (residual split by field
// between the two threads of a column, KS = 2), 4 = PAD (row pitch N+1),
// 8 = CONSTD (with SPLIT: t-derivative coefficients from the parameter bank; FP64),
// 16 = EARLY (without PIPE: neighbour traces requested before the tile wait),
// 32 = FACEFIRST (without PIPE: the face phase from global memory before the wait),
// 64 = DSMEM (with SPLIT: D rows from shared memory, fewer registers).
// ALG >= 1000: the bulk-copy one-tile form (stage_bulk.cuh: FP64, axis-aligned class)
// with second-family flags ALG - 1000 (SPLIT required; CONSTD; 16 = EARLY; 32 = KSM, k
// staged in shared memory by the bulk copies; DSMEM; 1 = ZCOL, tiles in z-column
// order on structured boxes; 4 = VROW, the r-derivative's rows read with 16-byte
// loads; 128 = ILP2, two partial sums per derivative; 256 / 512 = AHEAD, each block
// pulls into L2 the tile of the block half / one wave of resident blocks after it)
// and MINB resident blocks.  ALG 211 / 212: the field-split FP64 tensor-core tile with
// two warps per field (as 201) and that L2 pull half / one wave ahead.  ALG 2024 / 2056: the
// bulk-copy tile with four threads per column (stage_quad.cuh: FP64, axis-aligned class),
// k from L2 / staged in shared memory.
// Variant 0, the default, is entry 0 but at 9 points (NWB_DEFAULT): the fastest FP64 shape on
// B200 in a sweep of every shape over 8 M-node box meshes with fields in them.  The
// bulk-copy form leads everywhere but at 8 points, with the neighbour traces requested
// while the tile's copies fly (at 4 points four threads per column); k in shared memory but
// at 10 points, where it is read from L2 (the blocks that then fit pay more); the L2 pull
// only at 6 points.  A mesh of few elements takes another shape as its variant 0
// (NWB_SMALL), and there the number of that shape stands for the large default.  Per step, former default -> now: 90^3 of 2 points 2080 -> 1574 us, 62^3 of 3
// points 2218 -> 1545 us, 50^3 of 4 points 1569 -> 1405 us, 22^3 of 9 points 1500 -> 1337 us
// (there the pull and the z-column order had paid while the faces kept the L1 pipe busy),
// 20^3 of 10 points 1995 -> 1703 us.
// Variant numbers skip the FP64-only entries for FP32-bulk and for the other
// geometry classes, whose default is the first entry that is not FP64-only and
// which have that one variant.  The autotuner (nwb_solver_autotune) times every
// variant of the axis-aligned class on the caller's own mesh.  The pool's per-N
// kernels (batch.cu) use the same arithmetic as the default.
#pragma once

// The default of meshes with few elements: X(n, i), in order -- up to n elements variant 0
// is entry i of the list.  While a launch leaves SMs empty or is one or two waves of
// blocks, its time is that of one element's way through a block, which four threads
// per column halve; at 6 points one element per block instead of two fills the waves
// better up to 20 elements to an SM.  The lines lie where the times of both shapes
// cross on B200 (148 SMs), steps of n-element box meshes, default -> this shape: 64
// elements of 3 points 18.4 -> 12.3 us, 5 points 16.9 -> 14.4, 6 points 25.0 -> 17.4, 10
// points 52.8 -> 32.7; 2744 of 5 points 78.8 -> 71.7, 8000 of 5
// points 213.9 -> 213.2 (27000: 666 -> 695); 294 of 7 points 35.1 -> 28.7 (576: 46.0 -> 52.3);
// 125 of 9 points 42.0 -> 31.0 (150: 45.1 -> 52.3); 1100 of 10 points 288 -> 284 (1452: 353 ->
// 357); 1100 of 6 points 65.0 -> 54.2 (8000: 328 -> 355).  Not at 8 points (64 elements
// 27.7 -> 20.6): the tensor-core tile sums in another order, and a cavity's bits must not
// depend on what shares its launch; everywhere else all these shapes give the same bits.
#define NWB_SMALL_2(X) X(12 * 148, 4)
#define NWB_SMALL_3(X) X(14 * 148, 4)
#define NWB_SMALL_4(X)
#define NWB_SMALL_5(X) X(40 * 148, 25)
#define NWB_SMALL_6(X) X(2 * 148, 30) X(20 * 148, 29)
#define NWB_SMALL_7(X) X(2 * 148, 20)
#define NWB_SMALL_8(X)
#define NWB_SMALL_9(X) X(148, 19)
#define NWB_SMALL_10(X) X(8 * 148, 9)

// Index of the default's entry; that entry and entry 0 swap their variant numbers.  At 9
// points: X(2, 1, 0, 2, 1058), the bulk-copy tile with k in shared memory and neither pull
// nor z-column order.
#define NWB_DEFAULT(N) ((N) == 9 ? 13 : 0)

#define NWB_VARIANTS_2(X) X(2, 16, 0, 4, 1058) X(2, 16, 1, 1, 0) X(2, 32, 0, 2, 0) X(1, 32, 0, 2, 0) X(4, 8, 0, 4, 2056)
#define NWB_VARIANTS_3(X) X(2, 8, 0, 4, 1058) X(1, 16, 0, 4, 0) X(3, 8, 1, 1, 0) X(3, 8, 0, 3, 0) X(4, 2, 0, 8, 2056)
#define NWB_VARIANTS_4(X) X(4, 2, 0, 8, 2056) X(2, 4, 0, 4, 1026) X(2, 4, 0, 3, 13) X(2, 4, 0, 3, 5) X(1, 8, 0, 4, 0) X(2, 4, 1, 1, 0) X(2, 4, 0, 4, 0) X(4, 4, 0, 2, 0) X(2, 4, 0, 4, 4) X(2, 8, 0, 2, 4) X(2, 4, 0, 4, 12) X(2, 4, 0, 4, 20) X(2, 4, 0, 4, 28) X(2, 4, 0, 3, 1042) X(2, 4, 0, 3, 1058) X(2, 4, 0, 3, 1062)
#define NWB_VARIANTS_5(X) X(2, 1, 0, 8, 1058) X(2, 2, 0, 4, 1034) X(2, 2, 0, 5, 68) X(2, 2, 0, 4, 4) X(1, 4, 0, 4, 0) X(1, 4, 1, 1, 0) X(5, 2, 0, 2, 0) X(1, 8, 0, 2, 0) X(2, 4, 0, 2, 4) X(2, 2, 0, 4, 8) X(2, 2, 0, 4, 12) X(2, 2, 0, 5, 4) X(2, 2, 0, 4, 20) X(2, 2, 0, 4, 1050) X(2, 2, 0, 5, 1098) X(2, 2, 0, 4, 1035) X(2, 2, 0, 4, 1026) X(2, 2, 0, 5, 1058) X(2, 2, 0, 3, 1058) X(2, 2, 0, 4, 1058) X(2, 1, 0, 8, 1034) X(2, 2, 0, 4, 1062) X(2, 2, 0, 4, 1186) X(2, 1, 0, 8, 1314) X(2, 1, 0, 8, 1570) X(4, 1, 0, 6, 2056)
#define NWB_VARIANTS_6(X) X(2, 2, 0, 3, 1314) X(2, 2, 0, 3, 1058) X(2, 2, 0, 3, 1042) X(2, 2, 0, 3, 4) X(2, 2, 0, 3, 0) X(2, 2, 1, 1, 0) X(3, 2, 0, 2, 0) X(6, 1, 0, 2, 0) X(2, 4, 0, 1, 0) X(6, 1, 0, 3, 3) X(2, 2, 0, 3, 8) X(2, 2, 0, 3, 5) X(2, 2, 0, 3, 9) X(2, 4, 0, 2, 4) X(2, 2, 0, 3, 12) X(2, 2, 0, 3, 16) X(2, 2, 0, 4, 4) X(2, 2, 0, 5, 4) X(2, 4, 0, 2, 12) X(2, 2, 0, 3, 20) X(2, 2, 0, 3, 28) X(2, 2, 0, 3, 36) X(2, 2, 0, 3, 44) X(2, 2, 0, 3, 1034) X(2, 2, 0, 3, 1059) X(2, 2, 0, 3, 1062) X(2, 2, 0, 3, 1186) X(2, 2, 0, 3, 1570) X(2, 2, 0, 3, 1315) X(2, 1, 0, 5, 1058) X(4, 1, 0, 2, 2056)
#define NWB_VARIANTS_7(X) X(2, 1, 0, 4, 1058) X(2, 1, 0, 4, 1042) X(2, 1, 0, 4, 12) X(2, 1, 0, 4, 4) X(1, 2, 0, 3, 0) X(1, 2, 1, 1, 0) X(7, 1, 0, 2, 0) X(1, 4, 0, 1, 0) X(2, 2, 0, 3, 4) X(2, 2, 0, 3, 8) X(2, 1, 0, 5, 4) X(2, 1, 0, 6, 4) X(2, 1, 0, 4, 20) X(2, 1, 0, 3, 1042) X(2, 1, 0, 4, 1059) X(2, 1, 0, 4, 1026) X(2, 1, 0, 4, 1062) X(2, 1, 0, 4, 1186) X(2, 1, 0, 4, 1314) X(2, 1, 0, 4, 1570) X(4, 1, 0, 2, 2056)
#define NWB_VARIANTS_8(X) X(2, 1, 0, 4, 201) X(2, 1, 0, 4, 12) X(2, 1, 0, 4, 8) X(2, 1, 0, 4, 0) X(2, 1, 1, 1, 0) X(4, 1, 0, 2, 0) X(8, 1, 0, 1, 0) X(1, 2, 0, 2, 0) X(2, 2, 0, 2, 0) X(4, 1, 0, 2, 3) X(2, 1, 0, 4, 4) X(2, 1, 0, 3, 5) X(2, 1, 0, 3, 9) X(2, 1, 0, 4, 6) X(2, 1, 0, 4, 16) X(2, 1, 0, 4, 28) X(2, 1, 0, 4, 20) X(2, 1, 0, 4, 44) X(2, 1, 0, 4, 36) X(2, 1, 0, 3, 201) X(2, 1, 0, 3, 1) X(2, 1, 0, 3, 1042) X(2, 1, 0, 3, 1058) X(2, 1, 0, 3, 1062) X(2, 1, 0, 4, 211) X(2, 1, 0, 4, 212) X(4, 1, 0, 2, 2056)
#define NWB_VARIANTS_9(X) X(2, 1, 0, 2, 1315) X(2, 1, 0, 2, 1059) X(2, 1, 0, 2, 1042) X(2, 1, 0, 2, 12) X(2, 1, 0, 2, 4) X(3, 1, 0, 2, 0) X(1, 1, 1, 1, 0) X(1, 1, 0, 2, 0) X(9, 1, 0, 1, 0) X(2, 1, 0, 3, 4) X(2, 1, 0, 3, 8) X(2, 1, 0, 3, 12) X(2, 1, 0, 2, 1034) X(2, 1, 0, 2, 1058) X(2, 1, 0, 2, 1026) X(2, 1, 0, 2, 1062) X(2, 1, 0, 2, 1186) X(2, 1, 0, 2, 1571) X(2, 1, 0, 2, 1314) X(4, 1, 0, 1, 2056)
#define NWB_VARIANTS_10(X) X(2, 1, 0, 2, 1026) X(2, 1, 0, 2, 0) X(1, 1, 1, 1, 0) X(1, 1, 0, 2, 0) X(5, 1, 0, 1, 0) X(2, 1, 0, 3, 4) X(2, 1, 0, 3, 8) X(2, 1, 0, 2, 4) X(2, 1, 0, 2, 12) X(4, 1, 0, 1, 2024)
