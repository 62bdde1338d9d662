// A pred entry in 32 bits: the parent's id in the low PACK_BITS bits, the level
// above it, all ones = unreached.  Used where ids are below 2^PACK_BITS and levels
// at most PACK_MAX_LEVEL: level 31 with an all-ones parent would read as unreached.
#pragma once

#include <stdint.h>

namespace g500 {

constexpr int PACK_BITS = 27;
constexpr uint32_t PACK_ID = (1u << PACK_BITS) - 1u;
constexpr int PACK_MAX_LEVEL = 30;
constexpr uint32_t PACK_NONE = 0xFFFFFFFFu;

}  // namespace g500
