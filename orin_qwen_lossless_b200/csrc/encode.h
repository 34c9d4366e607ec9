// Host encoder of the BF16N format (see encode.cpp). Mirrors the reference's bf16n::encode (core/include/bf16n/encode.h:12-26).
#pragma once

#include "format.h"

#include <cstdint>
#include <functional>
#include <memory>
#include <utility>
#include <vector>

namespace b16 {

// Bytes that resize() leaves as the allocator gives them: the encoder writes every one of them, from all threads, and a
// zero fill beforehand would touch the pages of a large tensor once more, from one thread.
template <typename T> struct no_fill : std::allocator<T> {
    template <typename U> struct rebind { using other = no_fill<U>; };
    template <typename U> void construct(U * p) noexcept { ::new ((void *) p) U; }
    template <typename U, typename... A> void construct(U * p, A &&... a) { ::new ((void *) p) U(std::forward<A>(a)...); }
};
using Bytes = std::vector<uint8_t, no_fill<uint8_t>>;

struct Encoded {
    Bytes plane; // rows * K sign|mantissa bytes
    Bytes aux;   // 256-byte header + exponent data
    int format = 0;             // format produced (a HUFPAIR request falls back to HUFFMAN above 4096 distinct pairs)
    int R = 0;                  // rows per unit, 0 for NIBBLE
};

// rows x K BF16 bit patterns, row-major. Argument rules and std::invalid_argument behaviour as the reference:
//   NIBBLE: R = 0, no layout flags; HUFFMAN/HUFPAIR: R in {1,2,4,8,16}, rows % R == 0;
//   chunk_major: HUFPAIR, K > 512, R in {4,8,16}; frag_order: HUFPAIR, R = 16, not chunk-major; 512 <= K <= 4096, K % 512 == 0.
// plane: where the rows * K plane bytes go (null: into Encoded::plane). aux_memory: called once, with the number of aux bytes, for
// the memory they go to (empty: into Encoded::aux).
using AuxMemory = std::function<uint8_t *(size_t)>;
Encoded encode(const uint16_t * w, int64_t rows, int64_t K, int format, int R, bool chunk_major, bool frag_order = false,
               uint8_t * plane = nullptr, const AuxMemory & aux_memory = {});

} // namespace b16
