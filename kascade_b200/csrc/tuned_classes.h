// Size-class table: ruler spacing by a call's element count (KS_TUNED_SPACING:
// a batch, by its list elements; KS_TUNED_SPACING_SINGLE: one list) and
// chase block size.  Written by kascade_b200/autotune.py; the spacings from
// sweeps over 4 .. 80 at 3e4 .. 2.7e8 elements, e.g. lists of 2^20: 4 / 8 / 12
// / 24 157 / 164 / 152 / 193 us; 8e6: 8 / 16 / 32 556 / 530 / 582; 2^28: 24 /
// 32 / 48 / 64 13.9 / 13.7 / 13.4 / 13.4 ms; batches of 3e5
// elements: 4 / 6 / 8 / 16 137 / 131 / 141 / 160 us; 3e6: 6 / 8 / 16 / 24 259 /
// 250 / 270 / 291; 2e7: 8 / 16 / 24 976 / 903 / 912; 2^28: 24 / 32 / 40 10.6 /
// 10.6 / 10.5 ms.
#pragma once
#define KS_TUNED_GPU "NVIDIA B200"
#define KS_TUNED_COUNT 8
#define KS_TUNED_MAX {1024ull, 8192ull, 65536ull, 524288ull, 4194304ull, 33554432ull, 134217728ull, ~0ull}
#define KS_TUNED_SPACING {6u, 6u, 6u, 6u, 8u, 16u, 24u, 40u}
#define KS_TUNED_SPACING_SINGLE {4u, 4u, 6u, 6u, 12u, 16u, 32u, 48u}
#define KS_TUNED_CHAINS {1u, 1u, 1u, 1u, 1u, 1u, 4u, 4u}
#define KS_TUNED_BLOCK {256u, 128u, 128u, 512u, 512u, 256u, 256u, 256u}
