// chunkkey.h -- sort key that groups heavy rows by output chunk (batch.cu).
#pragma once

#include <cstdint>

#include "hd.h"

namespace gs {

// At most 2^20 uniform chunks and a cut after every doubling of the products at
// the boundaries of jobs that complete one by one.
constexpr int kChunkBits = 21;
constexpr int kChunkProdBits = 64 - kChunkBits - 1;

// By chunk, inside a chunk the windowed kernel's rows before the narrow rows,
// largest first (rows of more than 4e12 products among themselves in any order).
GS_HD uint64_t heavy_chunk_key(uint64_t chunk, bool narrow, uint64_t products) {
    constexpr uint64_t most = (1ull << kChunkProdBits) - 1;
    return (chunk << (kChunkProdBits + 1)) | ((uint64_t)narrow << kChunkProdBits) |
           (most - (products < most ? products : most));
}

}  // namespace gs
