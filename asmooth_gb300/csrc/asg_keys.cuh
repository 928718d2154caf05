// asg_keys.cuh -- a particle's key on the space-filling curve.
#pragma once

#include "asg_common.cuh"
#include "asg_internal.h"

namespace asg {

// space-filling-curve key, 16 bits per axis over [left, left + 65536 / scale)
__device__ __forceinline__ uint64_t space_key(const KeyGrid& g, float x, float y, float z)
{
    auto cell = [&](float c) -> uint32_t {
        float t = (c - g.left) * g.scale;
        t = fminf(fmaxf(t, 0.0f), 65535.0f);
        return (uint32_t)t;
    };
    const uint32_t cx = cell(x), cy = cell(y), cz = cell(z);
    return g.hilbert ? hilbert_key48(cx, cy, cz)
                     : spread3(cx) | (spread3(cy) << 1) | (spread3(cz) << 2);
}

}  // namespace asg
