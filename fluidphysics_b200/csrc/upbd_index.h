// Index arithmetic of the density pass's neighbour lists and chunks, right for
// every scene the library accepts (MAX_PARTICLES slots). Plain constexpr
// arithmetic with no CUDA types, so host code, device code and a CPU test
// compiled with g++ all see the same numbers.
#pragma once
#include "upbd_grid_layout.h"

namespace upbd {

constexpr long long MAX_PARTICLES = 1ll << 29;  // slots of a scene (check_desc)

constexpr int GLF = 4;       // lanes per particle of the fluid gathers
constexpr uint32_t NL = 28;  // list entries kept per lane (GLF * NL per particle)
constexpr uint32_t CHUNK = 32 / GLF;  // fluid particles of one cell that a warp takes

// Lane l's c-th entry is at row l * NL + c of a table with one column per slot:
// bytes from a column's first row. The row number stays far below 32 bits, a
// row's bytes are at most 2^31, their product does not (2^32 entries are reached from
// 38 million slots): one 32 x 32 -> 64 bit multiply.
UPBD_HD constexpr size_t list_row_bytes(uint32_t row, uint32_t slots) { return (size_t)row * (slots * 4u); }
static_assert(MAX_PARTICLES * 4 < (1ll << 32), "a list row's bytes are a 32-bit factor");

// A word of the chunk places: the size of the chunk that starts there (0: none)
// above the distance from the place to the particle's slot. Both lie in the
// particle's bucket, so the distance is below the bucket's size, which would
// have to pass 2^27 (the quadratic rank fix-up would never end) before it needs
// more bits than there are.
constexpr int CHUNK_SHIFT = 28;
UPBD_HD constexpr uint32_t chunk_word(uint32_t place, uint32_t slot, uint32_t size) {
  return ((slot - place) & ((1u << CHUNK_SHIFT) - 1u)) | (size << CHUNK_SHIFT);
}
UPBD_HD constexpr uint32_t chunk_word_size(uint32_t word) { return word >> CHUNK_SHIFT; }
UPBD_HD constexpr uint32_t chunk_word_slot(uint32_t place, uint32_t word) {
  return place + (uint32_t)((int32_t)(word << (32 - CHUNK_SHIFT)) >> (32 - CHUNK_SHIFT));
}
static_assert(CHUNK < (1u << (32 - CHUNK_SHIFT)), "a chunk's size fits above its distance");

// Groups of GL threads of the bond + contact pass (13 constraints a solid
// before them) and the displacement's DL threads a slot stay below 2^32.
constexpr int GL = 8;  // lanes per particle of the contact gathers and the solve
constexpr int DL = 2;  // threads per particle in the displacement pass
static_assert(MAX_PARTICLES * DL < (1ll << 32) && MAX_PARTICLES * (1 + 18 / GL + 1) < (1ll << 32),
              "32-bit numbers of threads and of lane groups");

}  // namespace upbd
