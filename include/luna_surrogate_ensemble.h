/*
 * The entry point of libluna_surrogate that the package's own predictions use beside those of
 * luna_surrogate.h (conventions as there).
 */
#ifndef LUNA_SURROGATE_ENSEMBLE_H
#define LUNA_SURROGATE_ENSEMBLE_H

#ifdef __cplusplus
extern "C" {
#endif

/* Last linear layer of an ensemble with its statistics, the members' outputs not written:
 * luna_sg_linear_fwd with act 0 into Yf, then luna_sg_ensemble, the same operations. mean [B x N]
 * (16-byte aligned) and spread [B] FP32. */
int luna_sg_linear_ensemble(const void* X, long long sX, const void* W, const float* b, int B, int K, int N, int nspec,
                            float* mean, float* spread, int members, int* err, void* stream);

#ifdef __cplusplus
}
#endif
#endif
