// Generated by ebbcfd_gb300/autotune.py on the default-size plate workload: device time per
// launch of each kernel of the three precision forms for each (threads per block) x (minimum
// resident blocks per SM requested through __launch_bounds__; 1 = the compiler's
// register choice), best of three rounds of CUDA-event timing.
// split k_cell: 64x12 136.8 us, 64x16 146.5 us, 128x6 137.6 us, 128x8 146.7 us, 128x10 165.0 us, 256x3 138.0 us, 256x4 149.5 us
// split k_flux: 64x16 120.1 us, 64x20 113.6 us, 128x8 120.8 us, 128x10 114.3 us, 128x12 106.6 us, 256x4 132.9 us, 256x6 109.4 us
// split k_update: 256x3 125.0 us, 256x4 129.3 us, 256x6 135.4 us, 256x8 174.8 us, 512x2 133.0 us, 512x3 133.9 us, 512x4 174.6 us
// fp64 k_cell: 64x12 2565.2 us, 64x16 2440.9 us, 128x6 2520.4 us, 128x8 2419.7 us, 128x10 2459.2 us, 256x3 2520.6 us, 256x4 2376.4 us
// fp64 k_flux: 64x6 2432.3 us, 64x8 2454.1 us, 128x1 2393.2 us, 128x4 2407.2 us, 128x5 2516.0 us, 128x6 2430.7 us, 256x2 2156.7 us
// fp64 k_update: 256x1 324.0 us, 256x2 323.9 us, 256x3 265.0 us, 256x4 253.6 us, 512x1 375.4 us, 512x2 262.8 us
// df k_cell: 64x12 795.6 us, 64x16 687.1 us, 128x6 803.5 us, 128x8 692.9 us, 128x10 645.1 us, 256x3 833.2 us, 256x4 714.6 us
// df k_flux: 64x6 558.5 us, 64x10 469.1 us, 128x4 498.3 us, 128x5 464.7 us, 128x6 472.8 us, 128x8 483.6 us, 256x2 541.1 us
// df k_update: 256x1 254.7 us, 256x2 254.7 us, 256x3 198.8 us, 256x4 190.4 us, 512x1 274.3 us, 512x2 198.9 us
// split_inv k_cell: 64x12 25.3 us, 64x16 24.1 us, 128x6 26.7 us, 128x8 24.6 us, 128x10 30.9 us, 256x3 27.2 us, 256x4 24.5 us
// split_inv k_flux: 64x16 24.8 us, 64x20 24.7 us, 128x8 20.8 us, 128x10 19.9 us, 128x12 18.5 us, 256x4 22.3 us, 256x6 18.6 us
// split_inv k_update: 256x4 31.4 us, 256x5 29.2 us, 256x6 29.3 us, 256x8 33.8 us, 512x2 31.7 us, 512x3 30.0 us, 512x4 38.6 us
// update block size 256 (summed best update times: 256: 598.3 us, 512: 624.7 us)
// The shapes below are the fastest of these rows but for FP64 k_cell, k_flux and k_update and
// double-float k_cell and k_update, which are as chosen on smaller plates (400,000 and 500,000
// cells: FP64 k_flux 128x4 194.7 us, 128x5 200.9, 128x6 202.2; k_update 256x3 32.6, 256x4 32.4;
// double-float k_update 256x3 28.0, 256x4 28.9); no other shape has been measured over the range
// of sizes.
#pragma once
#ifndef EBB_CELL_TB_F
#define EBB_CELL_TB_F 64
#endif
#ifndef EBB_CELL_MINB_F
#define EBB_CELL_MINB_F 12
#endif
#ifndef EBB_FLUX_TB_F
#define EBB_FLUX_TB_F 128
#endif
#ifndef EBB_FLUX_MINB_F
#define EBB_FLUX_MINB_F 12
#endif
#ifndef EBB_CELL4_TB_D
#define EBB_CELL4_TB_D 128
#endif
#ifndef EBB_CELL4_MINB_D
#define EBB_CELL4_MINB_D 8
#endif
#ifndef EBB_FLUX_TB_D
#define EBB_FLUX_TB_D 128
#endif
#ifndef EBB_FLUX_MINB_D
#define EBB_FLUX_MINB_D 4
#endif
#ifndef EBB_CELL4_TB_W
#define EBB_CELL4_TB_W 128
#endif
#ifndef EBB_CELL4_MINB_W
#define EBB_CELL4_MINB_W 8
#endif
#ifndef EBB_FLUX_TB_W
#define EBB_FLUX_TB_W 128
#endif
#ifndef EBB_FLUX_MINB_W
#define EBB_FLUX_MINB_W 5
#endif
#ifndef EBB_UPD_TB
#define EBB_UPD_TB 256
#endif
#ifndef EBB_UPD_MINB_F
#define EBB_UPD_MINB_F 3
#endif
#ifndef EBB_UPD_MINB_D
#define EBB_UPD_MINB_D 3
#endif
#ifndef EBB_UPD_MINB_W
#define EBB_UPD_MINB_W 3
#endif
#ifndef EBB_CELL_TB_FI
#define EBB_CELL_TB_FI 64
#endif
#ifndef EBB_CELL_MINB_FI
#define EBB_CELL_MINB_FI 16
#endif
#ifndef EBB_FLUX_TB_FI
#define EBB_FLUX_TB_FI 128
#endif
#ifndef EBB_FLUX_MINB_FI
#define EBB_FLUX_MINB_FI 12
#endif
#ifndef EBB_UPD_MINB_FI
#define EBB_UPD_MINB_FI 5
#endif
