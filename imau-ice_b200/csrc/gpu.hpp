// The GPU the kernels are sized for, in plain C++ (wave_geom.hpp is compiled for the CPU as well).
#pragma once

namespace diva {

constexpr int kSMs = 148;   // B200

}  // namespace diva
