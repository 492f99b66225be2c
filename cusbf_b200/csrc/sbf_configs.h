// sbf_configs.h -- the DNA configurations <K, S, M, H> whose kernels are compiled
// into the library (others are compiled at run time, sbf_jit.cpp).
#pragma once

// The benchmark configuration first; <31, s, 21, 4> is the reference's
// false-positive sweep over s (benchmarks/fpr_fastx_sweep.cu:294-302).
#define SBF_COMPILED_CONFIGS(X)                                                       \
    X(31, 28, 16, 4) X(31, 30, 16, 4) X(31, 31, 16, 4) X(31, 28, 16, 8) X(31, 28, 16, 16) \
    X(21, 19, 11, 4) X(5, 4, 3, 4) X(3, 2, 2, 4) X(31, 28, 21, 4) X(31, 30, 21, 4)     \
    X(31, 31, 21, 4)
