// Size-class table: mean ruler spacing by a call's list elements
// (KS_TUNED_SPACING: a batch's; KS_TUNED_SPACING_SINGLE: one list) and chase
// block size.  Chosen by hand from sweeps over 2 .. 80 at 3e4 .. 2.7e8 elements,
// one value for a class of sizes (us):
//   lists    2^18: 4 / 6 / 8 / 12 98 / 90 / 98 / 117
//            2^20: 4 / 6 / 8 / 12 / 16 134 / 128 / 125 / 150 / 146
//            2^21: 172 / 163 / 164 / 172 with 6 / 8 / 12 / 16
//            2^22: 285 / 256 / 237 / 231
//            8e6: 8 / 16 / 24 530 / 515 / 512
//            2^28: 24 / 32 / 48 / 64 13900 / 13700 / 13400 / 13400
//   batches  3e5: 4 / 6 / 8 / 16 137 / 131 / 141 / 160
//            3e6: 6 / 8 / 16 / 24 259 / 250 / 270 / 291
//            2e7: 8 / 16 / 24 976 / 903 / 912
//            2^28: 24 / 32 / 40 10600 / 10550 / 10530
// Classes up to 2^13 elements use no rulers, unless a call asks for a smaller
// one-CTA bound.  kascade_b200/autotune.py measures a table of this form for
// another GPU (tuning/b200.json is a run of it here) and can write this file.
#pragma once
#define KS_TUNED_GPU "NVIDIA B200"
#define KS_TUNED_COUNT 8
#define KS_TUNED_MAX {1024ull, 8192ull, 65536ull, 524288ull, 4194304ull, 33554432ull, 134217728ull, ~0ull}
#define KS_TUNED_SPACING {6u, 6u, 6u, 6u, 8u, 16u, 24u, 40u}
#define KS_TUNED_SPACING_SINGLE {4u, 4u, 6u, 6u, 12u, 16u, 32u, 48u}
#define KS_TUNED_CHAINS {1u, 1u, 1u, 1u, 1u, 1u, 1u, 1u}
#define KS_TUNED_BLOCK {256u, 128u, 128u, 512u, 512u, 256u, 256u, 256u}
