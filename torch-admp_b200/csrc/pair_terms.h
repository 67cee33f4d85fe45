// Pair-list energy launch shared by the entry points (pair_terms.cu).
#pragma once

#include "runtime.h"

namespace admp {

template <typename T>
int launch_pair_energy(int mode, int nf, int N, long long P, const long long* pairs, const T* ds, const void* bs,
                       bool int_scales, const T* q, const T* eta, double kappa, double ke, double* energy, int estride,
                       bool put, T* dds, T* dq, T* deta, DevError* err, cudaStream_t st);

}  // namespace admp
