// exact_shape.h -- compile-time shape constants of the exact kernel, shared by its host code.
#pragma once
#include <cstddef>
#include <cstdint>

namespace bude {

constexpr float kSteric = 76.f;   // 2 * HARDNESS (src/bude.h:33, serial/fasten.hpp:107)
constexpr int kClusterAtoms = 32; // protein atoms of one cluster: neighbours in space, tested lane by lane
constexpr int kPairF4 = 3;        // 16-byte words of the exact kernel's pair records
constexpr int kAtomAlign = 8;    // launch shapes name protein tiles in multiples of this
constexpr int kMaxThreads = 512; // threads of a block

} // namespace bude
