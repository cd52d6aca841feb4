// Constants of the fixed-point fluxes (fixed.cuh), set by the host.
#pragma once

namespace fvfix {

struct FluxConst {
    long long gamma;   // Q60: gamma * 2^60
    long long igm1_4;  // Q60: 2^60 / (4 (gamma - 1))
    float gammaf;
};

}  // namespace fvfix
