// Launch shapes of the hot kernels, chosen by teal_b200/autotune.py on a B200 (fastest measured RK
// step: TGV for the face, cell and gradient shapes, the ramp for the side-record face kernel, the ramp at
// space order 1 for the Euler staging switch and the Euler face occupancy; times within 0.5 % of the fastest
// count as ties, resolved to fewer resident face blocks, i.e. more registers per thread), and by single
// sweeps for the shapes it does not cover. Per launch at TGV 128^3: Navier-Stokes face 0.401 ms at 16
// blocks, 0.414 at 20, 0.445 at 12, 0.453 at 24; FP32-flux face 0.309 ms at 32 blocks against 0.326 at 20;
// gradient 0.264 against 0.280 ms at 9 (both before its tiles). A step of the ramp of 513 k cells: 401 us with
// the side-record face kernel at 6 blocks, 402 at 7, 403 at 8, 414 at 5 (64-thread blocks 400, 256-thread
// ones 407); at space order 1 221 us staged at 28 blocks, 224 not staged, 223 at 24 or 32, 228 at 20. A value
// given with -D at build time wins.
#pragma once

#ifndef TG_FACE_BLOCK
#define TG_FACE_BLOCK 32  // threads per face-flux block
#endif
#ifndef TG_FACE_MINB
#define TG_FACE_MINB 16  // Navier-Stokes face-flux blocks kept resident per SM (caps registers per thread)
#endif
#ifndef TG_FACE_MINB_FP32
#define TG_FACE_MINB_FP32 32  // FP32-flux face-flux blocks kept resident per SM (caps registers per thread)
#endif
#ifndef TG_FACE_MINB_EULER
#define TG_FACE_MINB_EULER 28  // first-order and exact Euler face-flux blocks kept resident per SM (caps registers per thread)
#endif
#ifndef TG_SIDE_BLOCK
#define TG_SIDE_BLOCK 128  // threads per face-flux block between side records
#endif
#ifndef TG_SIDE_MINB
#define TG_SIDE_MINB 6  // its blocks kept resident per SM, FP64
#endif
#ifndef TG_SIDE_MINB_FP32
#define TG_SIDE_MINB_FP32 8  // its blocks kept resident per SM, FP32-flux form
#endif
#ifndef TG_FUSED_CELLS
#define TG_FUSED_CELLS 18944  // most cells of an arena whose face fluxes and cell updates run in one launch (148 x 128)
#endif
#ifndef TG_CELL_BLOCK
#define TG_CELL_BLOCK 128  // threads per cell-gather block
#endif
#ifndef TG_FACE_STAGED_EULER
#define TG_FACE_STAGED_EULER 1  // first-order and exact Euler face kernel: geometry staged by bulk copies (1) or loaded (0)
#endif
#ifndef TG_CELL_MINB
#define TG_CELL_MINB 10  // cell-gather blocks kept resident per SM (caps registers per thread)
#endif
#ifndef TG_CELL_MINB_RESIDUAL
#define TG_CELL_MINB_RESIDUAL 8  // the same for a bare residual (derivative calls, implicit steps)
#endif
#ifndef TG_CELL_MINB_FP32
#define TG_CELL_MINB_FP32 12  // the same in the FP32-flux form
#endif
#ifndef TG_GRAD_MINB
#define TG_GRAD_MINB 12  // gradient blocks (160 threads) kept resident per SM (caps registers per thread)
#endif
#ifndef TG_GRAD_MINB_SIDES
#define TG_GRAD_MINB_SIDES 9  // the same for the gradient kernel that writes side records
#endif
