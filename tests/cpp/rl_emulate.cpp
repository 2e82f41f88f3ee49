// CPU emulation of k_sweep_rl on the row words, in-chain columns and entries that
// the layout builder (wf_layout.hpp, chain-major) makes: every index of the
// kernel checked, a gathered row must belong to an earlier colour, an in-chain
// column to a row of the chain solved before; the rows of a chain are recomputed
// together as often as the chain has levels. Test code only.
#include <cstdio>

#include "wf_layout.hpp"

using namespace senkgpu;

namespace {

// info[0]: words per row (0: the builder refused the chain-major layout)
template <typename VT>
int emulate(int N, const VT *val, const int *cind, const int *rptr, int upper, const int *cptr, int cnum, int bs,
            const VT *x, VT *y, int *info, char *err, int errlen)
{
    auto fail = [&](const char *m, int row) {
        std::snprintf(err, errlen, "%s (row %d)", m, row);
        return 1;
    };
    try {
        std::vector<WfColour> colours;
        std::vector<int> colour_of(N);
        for (int k = 0; k < cnum; k++) {
            const int c = upper ? cnum - 1 - k : k;
            colours.push_back({cptr[c] * bs, cptr[c + 1] * bs});
            for (int p = cptr[c] * bs; p < cptr[c + 1] * bs; p++) colour_of[p] = k;
        }
        WfLayout<VT> L;
        info[0] = 0;
        if (!make_wf_layout(L, upper != 0, N, val, cind, rptr, colours, bs, colour_of.data(), (size_t)1 << 30, nullptr,
                            true))
            return 0;
        const size_t ng = L.groups.size();
        const int rw = (int)(L.rows.size() / (ng * 32 * bs));
        if ((rw != 1 && rw != 2) || L.rows.size() != ng * 32 * bs * rw) return fail("row words", -1);
        info[0] = rw;
        std::vector<VT> yy(x, x + N);
        std::vector<int> done(N, 0);
        for (size_t k = 0; k + 1 < L.colour_groups.size(); k++) {
            std::vector<int> fin;
            std::vector<VT> res;
            for (int g = L.colour_groups[k]; g < L.colour_groups[k + 1]; g++) {
                const WfGroup d = L.groups[g];
                const int *cw = L.col.data() + d.off;
                const VT *vw = L.val.data() + d.off, *iv = vw + (size_t)d.emax * 32;
                const unsigned char *ic = L.icol.data() + d.off + (size_t)d.emax * 32;
                for (int q = 0; q < d.nchains; q++) {
                    const int2 cd = L.chains[(size_t)g * 32 + q];
                    const int r0 = cd.x, ib = (int)((unsigned)cd.y >> 16);
                    std::vector<VT> t(bs), out(bs);
                    std::vector<RowWord> u(bs);
                    for (int rr = 0; rr < bs; rr++) {
                        const unsigned *w = &L.rows[(((size_t)g * 32 + q) * bs + rr) * rw];
                        u[rr] = rw == 2 ? row_word(make_uint2(w[0], w[1])) : row_word(w[0]);
                        const int row = r0 + rr;
                        int ext = 0, in = 0;
                        for (int j = rptr[row] + (upper ? 1 : 0); j < rptr[row + 1]; j++)
                            (cind[j] >= r0 && cind[j] < r0 + bs ? in : ext)++;
                        if (u[rr].ne != ext || u[rr].left != in) return fail("counts of a row", row);
                        t[rr] = yy[row];
                        for (int e = 0; e < u[rr].ne; e++) {
                            const int at = u[rr].eo + e;
                            if (at >= d.emax) return fail("external entry beyond the chain's stream", row);
                            const int c = cw[(size_t)q * d.emax + at] & kColMask;
                            if (c < 0 || c >= N || !done[c]) return fail("gathers a row that is not finished", row);
                            t[rr] -= vw[(size_t)q * d.emax + at] * yy[c];
                        }
                        for (int e = 0; e < u[rr].left; e++) {
                            const int at = ib + u[rr].io + e;
                            if (at >= d.imax * 32) return fail("in-chain entry beyond the block", row);
                            if (upper ? ic[at] <= rr : ic[at] >= rr) return fail("in-chain column out of order", row);
                            if (ic[at] >= bs) return fail("in-chain column out of the chain", row);
                        }
                        out[rr] = upper ? t[rr] * L.dinv[row] : t[rr];
                    }
                    for (int l = 0; l < u[0].depth; l++) {
                        const std::vector<VT> before(out);
                        for (int rr = 0; rr < bs; rr++) {
                            VT a = t[rr];
                            for (int e = 0; e < u[rr].left; e++)
                                a -= iv[ib + u[rr].io + e] * before[ic[ib + u[rr].io + e]];
                            out[rr] = upper ? a * L.dinv[r0 + rr] : a;
                        }
                    }
                    for (int rr = 0; rr < bs; rr++) {
                        fin.push_back(r0 + rr);
                        res.push_back(out[rr]);
                    }
                }
            }
            for (size_t i = 0; i < fin.size(); i++) {
                yy[fin[i]] = res[i];
                done[fin[i]] = 1;
            }
        }
        std::copy(yy.begin(), yy.end(), y);
        return 0;
    } catch (const std::exception &e) {
        std::snprintf(err, errlen, "%s", e.what());
        return 1;
    }
}

}  // namespace

extern "C" int rl_emulate_d(int N, const double *val, const int *cind, const int *rptr, int upper, const int *cptr,
                            int cnum, int bs, const double *x, double *y, int *info, char *err, int errlen)
{
    return emulate(N, val, cind, rptr, upper, cptr, cnum, bs, x, y, info, err, errlen);
}

extern "C" int rl_emulate_s(int N, const float *val, const int *cind, const int *rptr, int upper, const int *cptr,
                            int cnum, int bs, const float *x, float *y, int *info, char *err, int errlen)
{
    return emulate(N, val, cind, rptr, upper, cptr, cnum, bs, x, y, info, err, errlen);
}
