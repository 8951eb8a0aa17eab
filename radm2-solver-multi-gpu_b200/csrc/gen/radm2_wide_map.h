/* Generated by radm2-solver-multi-gpu_b200/mech/emit_wide.py from mech/radm2_mech.json
 * (the RADM2 mechanism as encoded in the reference's mgpu.cu).  Do not edit. */
#pragma once
/* Working-set placement of the wide tensor-memory solver, in doubles per thread: RC_WORDS
 * distinct rate constants (word k holds the constant of reaction RC_REP[k]; the 68 others are
 * numbers or repeats); LU slots by their loads and stores per step attempt: 256 in tensor memory
 * (2980 of 5384 accesses), 79 in shared memory (600), 324 in global scratch (1804). */
#define RADM2_WIDE_RC_WORDS 88
#define RADM2_WIDE_RC_REP_INIT {0,1,2,3,4,5,6,7,8,9,10,11,12,13,14,15,16,17,18,19,20,21,22,23,25,26,27,28,29,30,31,32,33,34,35,36,37,38,40,41,42,43,44,45,46,47,48,49,50,51,52,53,54,55,56,57,58,61,62,69,70,71,72,73,76,90,91,96,97,98,100,101,102,103,104,118,119,120,121,122,125,127,131,132,133,134,139,146}
#define RADM2_WIDE_SMEM_WORDS 226
#define RADM2_WIDE_GLOBAL_WORDS 501
#define RADM2_WIDE_GRCP 501   /* division form: 59 more words, the reciprocal pivots */
#define RADM2_WIDE_GLOBAL_WORDS_DIV 560
#define RADM2_WIDE_SPIVOT 147   /* the 28 pivots of rows without eliminations, side by side */
#define RADM2_WIDE_SPIVOTS 28
#define RADM2_WIDE_GK1 0
#define RADM2_WIDE_GK2 59
#define RADM2_WIDE_GY 118
