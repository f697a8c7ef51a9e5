// residual2_tuned.h -- written by autotune.py: the fastest candidate per degree on this GPU
// (residual ms per launch, vortex mesh of about 33 M DOFs; set 0 stays unless another is faster by more
// than 1 %).
//   p=1 MHD_RES2_CFG (4, 2, 32, 16): 0.1653 ms  <- chosen
//   p=1 MHD_RES2_CFG (4, 4, 64, 8): 0.1672 ms
//   p=1 MHD_RES2_CFG (8, 4, 128, 4): 0.1727 ms
//   p=1 MHD_RES2_CFG (4, 2, 32, 18): 0.1827 ms
#ifndef MHD_RES2_CFG1
#define MHD_RES2_CFG1 4, 2, 32, 16
#endif
//   p=2 MHD_RES2_CFG (3, 1, 32, 16): 0.1790 ms  <- chosen
//   p=2 MHD_RES2_CFG (3, 2, 64, 8): 0.1808 ms
//   p=2 MHD_RES2_CFG (6, 2, 128, 4): 0.1839 ms
//   p=2 MHD_RES2_CFG (3, 1, 32, 18): 0.2064 ms
#ifndef MHD_RES2_CFG2
#define MHD_RES2_CFG2 3, 1, 32, 16
#endif
//   p=3 MHD_RES2_CFG (2, 1, 32, 16): 0.2750 ms  <- chosen
//   p=3 MHD_RES2_CFG (2, 2, 64, 8): 0.2750 ms
//   p=3 MHD_RES2_CFG (4, 2, 128, 4): 0.2783 ms
//   p=3 MHD_RES2_CFG (2, 1, 32, 17): 0.3083 ms
#ifndef MHD_RES2_CFG3
#define MHD_RES2_CFG3 2, 1, 32, 16
#endif
