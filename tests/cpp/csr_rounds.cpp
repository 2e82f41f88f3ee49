// CPU walk of k_spmv_csr_rows' tiles and rounds (csr_rounds.hpp), as the kernel
// makes them: every copied piece and every row's share of a round is checked
// against the arrays' ends and the rows. Test code only.
#include <algorithm>
#include <cstdio>

#include "csr_rounds.hpp"

using namespace senkgpu;

// The tile `tile` of an n-row matrix with nnz entries whose rows have the ends
// rp[0..32] (the tile's part of the row pointer; rows past n repeat the last).
extern "C" int csr_walk(int n, int nnz, int tile, const int *rp, int cap, int size, char *err, int errlen)
{
    auto fail = [&](const char *m, long long v) {
        std::snprintf(err, errlen, "%s (%lld)", m, v);
        return 1;
    };
    const int tiles = csr_tiles(n), EV = 16 / size;
    if ((long long)tiles * 32 < n || (long long)(tiles - 1) * 32 >= n) return fail("tiles do not cover the rows", tiles);
    int a[32], e[32];
    for (int lane = 0; lane < 32; lane++) {
        const int r = tile * 32 + lane;
        const long long b = csr_begin_at(r, n), t = csr_end_at(r, n);
        if (r < 0 || b != std::min<long long>((long long)tile * 32 + lane, n) ||
            t != std::min<long long>((long long)tile * 32 + lane + 1, n))
            return fail("row pointer out of range", r);
        a[lane] = rp[b - (long long)tile * 32];
        e[lane] = rp[t - (long long)tile * 32];
    }
    int c0 = a[0] & ~3;
    const int s1 = e[31];
    long long done[32] = {};
    for (long long rounds = 0;; rounds++) {
        if (rounds > 1000000) return fail("does not end", c0);
        const int cnt = csr_round(c0, cap, s1);
        if (cnt > cap) return fail("more entries than the buffer holds", cnt);
        for (int width : {size, 4})
            for (int i = 0; i < cnt; i += 16 / width) {
                const long long at = (long long)c0 + i, bytes = csr_piece_bytes(c0 + i, nnz, width);
                if (at % (16 / width)) return fail("misaligned piece", at);
                // exactly the entries of the piece that the array has
                if (bytes != std::min<long long>(16, (nnz - at) * width)) return fail("wrong bytes of a piece", bytes);
                if (bytes <= 0 || bytes > 16) return fail("a copy of this many bytes", bytes);
            }
        for (int lane = 0; lane < 32; lane++) {
            const int lo = std::max(a[lane] - c0, 0), len = std::min(e[lane] - c0, cap) - lo;
            for (int f = 0; f < len; f++)
                if (lo + f >= (cnt + EV - 1) / EV * EV || (long long)c0 + lo + f != a[lane] + done[lane]++)
                    return fail("a row's entry that was not staged", (long long)c0 + lo + f);
        }
        if (!csr_more(c0, cap, s1)) break;
        c0 += cap;
    }
    for (int lane = 0; lane < 32; lane++)
        if (done[lane] != e[lane] - a[lane]) return fail("entries left out of a row", lane);
    return 0;
}
