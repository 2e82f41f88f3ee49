// Index arithmetic of k_spmv_csr_rows, for rows and entries over the whole range
// of int: tiles of 32 rows, and the rounds of `cap` entries in which a tile's
// entries are staged. Plain code, so that it runs on the host too.
#pragma once

#ifndef SENK_HD
#ifdef __CUDACC__
#define SENK_HD __host__ __device__
#else
#define SENK_HD
#endif
#endif

namespace senkgpu {

// Tiles of n rows.
SENK_HD constexpr int csr_tiles(int n) { return (int)(((unsigned)n + 31u) >> 5); }

// Where row pointer r and the one after it stand, for a row that may lie past n.
SENK_HD constexpr int csr_begin_at(int r, int n) { return r < n ? r : n; }
SENK_HD constexpr int csr_end_at(int r, int n) { return r < n ? r + 1 : n; }

// Bytes to copy of the 16-byte piece that starts at entry `at` of nnz (at < nnz),
// entries of `size` bytes: the entries left are compared, not their bytes, which
// pass 2^31 from 2^28 entries of 8 bytes on.
SENK_HD constexpr int csr_piece_bytes(int at, int nnz, int size)
{
    const int left = nnz - at;
    return left >= 16 / size ? 16 : left * size;
}

// Whether a tile that ends at entry s1 has entries past the round from c0, and
// how many this round holds (c0 + cap may lie past the range).
SENK_HD constexpr bool csr_more(int c0, int cap, int s1) { return s1 - c0 > cap; }
SENK_HD constexpr int csr_round(int c0, int cap, int s1) { return s1 - c0 < cap ? s1 - c0 : cap; }

}  // namespace senkgpu
