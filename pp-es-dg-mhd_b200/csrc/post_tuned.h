// post_tuned.h -- written by autotune.py: the fastest candidate per degree on this GPU
// (ms per SSP-RK3 step (OEDG + LDF + PP), vortex mesh of about 33 M DOFs; set 0 stays unless another is faster by more
// than 1 %).
//   p=1 MHD_PP_CFG (256, 4); MHD_SIG_CFG (16, 4, 4): 0.8919 ms  <- chosen
//   p=1 MHD_PP_CFG (256, 4); MHD_SIG_CFG (8, 8, 4): 0.8973 ms
//   p=1 MHD_PP_CFG (256, 4); MHD_SIG_CFG (8, 8, 5): 0.8989 ms
//   p=1 MHD_PP_CFG (128, 8); MHD_SIG_CFG (16, 4, 4): 0.8928 ms
#ifndef MHD_PP_CFG1
#define MHD_PP_CFG1 256, 4
#endif
#ifndef MHD_SIG_CFG1
#define MHD_SIG_CFG1 16, 4, 4
#endif
//   p=2 MHD_PP_CFG (256, 4); MHD_SIG_CFG (8, 4, 5): 1.0566 ms  <- chosen
//   p=2 MHD_PP_CFG (256, 4); MHD_SIG_CFG (8, 4, 4): 1.0609 ms
//   p=2 MHD_PP_CFG (256, 4); MHD_SIG_CFG (4, 4, 6): 1.0763 ms
//   p=2 MHD_PP_CFG (128, 8); MHD_SIG_CFG (8, 4, 5): 1.0561 ms
#ifndef MHD_PP_CFG2
#define MHD_PP_CFG2 256, 4
#endif
#ifndef MHD_SIG_CFG2
#define MHD_SIG_CFG2 8, 4, 5
#endif
//   p=3 MHD_PP_CFG (256, 4); MHD_SIG_CFG (4, 4, 4): 1.5050 ms  <- chosen
//   p=3 MHD_PP_CFG (256, 4); MHD_SIG_CFG (4, 4, 3): 1.5233 ms
//   p=3 MHD_PP_CFG (256, 4); MHD_SIG_CFG (2, 8, 4): 1.5204 ms
//   p=3 MHD_PP_CFG (128, 8); MHD_SIG_CFG (4, 4, 4): 1.5030 ms
#ifndef MHD_PP_CFG3
#define MHD_PP_CFG3 256, 4
#endif
#ifndef MHD_SIG_CFG3
#define MHD_SIG_CFG3 4, 4, 4
#endif
