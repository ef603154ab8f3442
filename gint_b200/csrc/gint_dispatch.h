/*
 * gint_dispatch.h -- the jump tables of the interpreter's dispatch as PTX text, for inline assembly (gint_interp.cuh).
 *
 * Handler labels are GL<depth>_<opcode>. GINT_BRANCH_TABLES declares one table GT<depth> per stack depth, over the opcodes the
 * kernel family dispatches on (rounded up to a multiple of ten, GINT_N_TABLE); GINT_BRANCH_TABLE_ALL declares one table GTALL
 * over every key depth * GINT_N_TABLE + opcode. Every label of a table is defined in the kernel, by a handler or in the
 * default block.
 */
#ifndef GINT_DISPATCH_H
#define GINT_DISPATCH_H

#include "gint_opcodes.h"

#define GINT_N_TABLE ((GINT_N_DISPATCH + 9) / 10 * 10)
#define GINT_N_KEYS ((GINT_MAX_STACK + 1) * GINT_N_TABLE)

#define GINT_L(d, n) "GL" #d "_" #n
/* ten labels: opcodes t0 .. t9 (t empty: 0 .. 9) */
#define GINT_L10(d, t)                                                                                                  \
    GINT_L(d, t##0) ", " GINT_L(d, t##1) ", " GINT_L(d, t##2) ", " GINT_L(d, t##3) ", " GINT_L(d, t##4) ", "              \
    GINT_L(d, t##5) ", " GINT_L(d, t##6) ", " GINT_L(d, t##7) ", " GINT_L(d, t##8) ", " GINT_L(d, t##9)
#define GINT_L150(d)                                                                                                     \
    GINT_L10(d, ) ",\n\t" GINT_L10(d, 1) ",\n\t" GINT_L10(d, 2) ",\n\t" GINT_L10(d, 3) ",\n\t" GINT_L10(d, 4) ",\n\t"       \
    GINT_L10(d, 5) ",\n\t" GINT_L10(d, 6) ",\n\t" GINT_L10(d, 7) ",\n\t" GINT_L10(d, 8) ",\n\t" GINT_L10(d, 9) ",\n\t"      \
    GINT_L10(d, 10) ",\n\t" GINT_L10(d, 11) ",\n\t" GINT_L10(d, 12) ",\n\t" GINT_L10(d, 13) ",\n\t" GINT_L10(d, 14)
#if defined(GINT_RF)
#define GINT_LABELS(d) GINT_L150(d) ",\n\t" GINT_L10(d, 15) ",\n\t" GINT_L10(d, 16) ",\n\t" GINT_L10(d, 17)
#elif defined(GINT_VEC)
#define GINT_LABELS(d) GINT_L150(d) ",\n\t" GINT_L10(d, 15) ",\n\t" GINT_L10(d, 16) ",\n\t" GINT_L10(d, 17) ",\n\t" GINT_L10(d, 18)
#else
#define GINT_LABELS(d) GINT_L150(d)
#endif

#define GINT_TABLE(d) "GT" #d ": .branchtargets\n\t" GINT_LABELS(d) ";\n\t"
#define GINT_BRANCH_TABLES                                                                                               \
    GINT_TABLE(0) GINT_TABLE(1) GINT_TABLE(2) GINT_TABLE(3) GINT_TABLE(4) GINT_TABLE(5) GINT_TABLE(6) GINT_TABLE(7) GINT_TABLE(8)
#define GINT_BRANCH_TABLE_ALL                                                                                            \
    "GTALL: .branchtargets\n\t" GINT_LABELS(0) ",\n\t" GINT_LABELS(1) ",\n\t" GINT_LABELS(2) ",\n\t" GINT_LABELS(3) ",\n\t"  \
    GINT_LABELS(4) ",\n\t" GINT_LABELS(5) ",\n\t" GINT_LABELS(6) ",\n\t" GINT_LABELS(7) ",\n\t" GINT_LABELS(8) ";\n\t"

/* The streaming kernels have two tables per depth (0 .. 4), outside of loops GTN<depth> (opcodes 0 .. 129) and inside GTW<depth>
 * (from GINT_WIDE_TABLE_FIRST = 100 on): half the edges in the control-flow graph. */
#define GINT_LABELS_NARROW(d)                                                                                            \
    GINT_L10(d, ) ",\n\t" GINT_L10(d, 1) ",\n\t" GINT_L10(d, 2) ",\n\t" GINT_L10(d, 3) ",\n\t" GINT_L10(d, 4) ",\n\t"       \
    GINT_L10(d, 5) ",\n\t" GINT_L10(d, 6) ",\n\t" GINT_L10(d, 7) ",\n\t" GINT_L10(d, 8) ",\n\t" GINT_L10(d, 9) ",\n\t" GINT_L10(d, 10) ",\n\t"     \
    GINT_L10(d, 11) ",\n\t" GINT_L10(d, 12)
#define GINT_LABELS_WIDE(d)                                                                                              \
    GINT_L10(d, 10) ",\n\t" GINT_L10(d, 11) ",\n\t" GINT_L10(d, 12) ",\n\t" GINT_L10(d, 13) ",\n\t" GINT_L10(d, 14) ",\n\t"  \
    GINT_L10(d, 15) ",\n\t" GINT_L10(d, 16) ",\n\t" GINT_L10(d, 17) ",\n\t" GINT_L10(d, 18) ",\n\t" GINT_L10(d, 19) ",\n\t"  \
    GINT_L10(d, 20) ",\n\t" GINT_L10(d, 21) ",\n\t" GINT_L10(d, 22) ",\n\t" GINT_L10(d, 23)
#define GINT_TABLE_PAIR(d) "GTN" #d ": .branchtargets\n\t" GINT_LABELS_NARROW(d) ";\n\tGTW" #d ": .branchtargets\n\t" GINT_LABELS_WIDE(d) ";\n\t"
#define GINT_WIDE_BRANCH_TABLES GINT_TABLE_PAIR(0) GINT_TABLE_PAIR(1) GINT_TABLE_PAIR(2) GINT_TABLE_PAIR(3) GINT_TABLE_PAIR(4)

#endif /* GINT_DISPATCH_H */
