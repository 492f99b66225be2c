// sbf_narrow.cuh -- table of the tile kernels with strips of `Strip` windows.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "sbf_configs.h"
#include "sbf_internal.h"
#include "sbf_tile.cuh"

namespace sbf {

template <class C>
const void* narrow_variant(int which) {
    const void* const fns[6] = {
        reinterpret_cast<const void*>(&tile_kernel<C, false, false, false>),
        reinterpret_cast<const void*>(&tile_kernel<C, true, false, false>),
        reinterpret_cast<const void*>(&tile_kernel<C, false, true, false>),
        reinterpret_cast<const void*>(&tile_kernel<C, true, true, false>),
        reinterpret_cast<const void*>(&tile_kernel<C, false, false, true>),
        reinterpret_cast<const void*>(&tile_kernel<C, true, false, true>)};
    return fns[which];
}

// Kernel `which` (KernelSet order) of the config-th compiled configuration.
template <int Strip>
const void* narrow_kernel_of(int config, int which) {
    int i = 0;
#define SBF_NARROW(K, S, M, H) \
    if (config == i++) return narrow_variant<Cfg<K, S, M, H, Strip>>(which);
    SBF_COMPILED_CONFIGS(SBF_NARROW)
#undef SBF_NARROW
    return nullptr;
}

}  // namespace sbf
