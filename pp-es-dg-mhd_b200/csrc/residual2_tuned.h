// residual2_tuned.h -- written by autotune.py: the fastest candidate per degree on this GPU
// (residual ms per launch, vortex mesh of about 33 M DOFs; set 0 stays unless another is faster by more
// than 1 %).
//   p=1 MHD_RES2_CFG (4, 2, 32, 16): 0.1642 ms  <- chosen
//   p=1 MHD_RES2_CFG (4, 4, 64, 8): 0.1669 ms
//   p=1 MHD_RES2_CFG (8, 4, 128, 4): 0.1689 ms
//   p=1 MHD_RES2_CFG (4, 2, 32, 18): 0.1829 ms
#ifndef MHD_RES2_CFG1
#define MHD_RES2_CFG1 4, 2, 32, 16
#endif
//   p=2 MHD_RES2_CFG (3, 1, 32, 16): 0.1754 ms  <- chosen
//   p=2 MHD_RES2_CFG (3, 2, 64, 8): 0.1785 ms
//   p=2 MHD_RES2_CFG (6, 2, 128, 4): 0.1818 ms
//   p=2 MHD_RES2_CFG (3, 1, 32, 18): 0.2012 ms
#ifndef MHD_RES2_CFG2
#define MHD_RES2_CFG2 3, 1, 32, 16
#endif
//   p=3 MHD_RES2_CFG (2, 1, 32, 16): 0.2745 ms  <- chosen
//   p=3 MHD_RES2_CFG (2, 2, 64, 8): 0.2725 ms
//   p=3 MHD_RES2_CFG (4, 2, 128, 4): 0.2756 ms
//   p=3 MHD_RES2_CFG (2, 1, 32, 17): 0.3089 ms
#ifndef MHD_RES2_CFG3
#define MHD_RES2_CFG3 2, 1, 32, 16
#endif
