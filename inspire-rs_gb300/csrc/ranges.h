// ranges.h -- conditions on a caller's host buffers that kernels read and
// write in place, kept free of CUDA so that a host-only check (tests/native)
// can exercise them.  Internal; not part of the public header.
#pragma once
#include <cstddef>
#include <cstdint>

namespace ighost {

inline bool aligned(const void* p, size_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; }

// Whether [a, a + na) and [b, b + nb) share a byte.  A kernel that answers one
// query while another's rows are still to be read must not write where they lie.
inline bool overlap(const void* a, size_t na, const void* b, size_t nb) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return na && nb && (x < y ? y - x < na : x - y < nb);
}

// Whether a batch's rows may be read and its responses written in place: rows
// 16-byte aligned (they are bulk-copied), responses where 64-bit words may be
// stored, and apart from the rows.
inline bool rows_and_out_in_place(const void* rows, size_t rows_bytes, const void* out, size_t out_bytes) {
  return aligned(rows, 16) && aligned(out, sizeof(uint64_t)) && !overlap(rows, rows_bytes, out, out_bytes);
}

}  // namespace ighost
