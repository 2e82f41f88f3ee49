// CPU emulation of the slice sweep (k_sweep_lv) on the layout that the plan
// builds (senk_gb300/csrc/lv_layout.hpp): every access of the kernel with its
// index checked, colour by colour; a gathered row must belong to an earlier
// colour, an in-chain row to an earlier level of its group. Test code only.
#include <cstdio>

#include "lv_layout.hpp"

using namespace senkgpu;

namespace {

template <typename VT>
int emulate(int N, const VT *val, const int *cind, const int *rptr, int upper, const int *cptr, int cnum, int bs,
            int want, int spread, const VT *x, VT *y, int *info, char *err, int errlen)
{
    auto fail = [&](const char *m) {
        std::snprintf(err, errlen, "%s", m);
        return 1;
    };
    try {
        std::vector<std::pair<int, int>> colours;
        std::vector<int> colour_of(N);
        for (int k = 0; k < cnum; k++) {
            const int c = upper ? cnum - 1 - k : k;
            colours.push_back({cptr[c] * bs, cptr[c + 1] * bs});
            for (int p = cptr[c] * bs; p < cptr[c + 1] * bs; p++) colour_of[p] = k;
        }
        LvLayout<VT> L;
        if (!make_lv_layout(L, upper != 0, N, val, cind, rptr, colours, bs, colour_of.data(), (size_t)want, spread,
                            (size_t)1 << 30))
            return fail("layout does not fit");
        info[0] = *std::min_element(L.colour_rows.begin(), L.colour_rows.end());
        std::vector<VT> yy(x, x + N);
        std::vector<int> done(N, 0);
        long long stored = 0;
        for (size_t k = 0; k + 1 < L.colour_groups.size(); k++) {
            std::vector<VT> next(yy);
            for (int g = L.colour_groups[k]; g < L.colour_groups[k + 1]; g++) {
                const LvGroup d = L.groups[g];
                const unsigned char *t = L.blocks.get() + (size_t)d.off * 16;
                const LvHeader *h = (const LvHeader *)t;
                const LvParts P = lv_parts(*h, upper ? d.nrows * (unsigned)sizeof(VT) : 0u, sizeof(VT));
                if (d.nrows < 1 || d.nrows > L.colour_rows[k] || P.end != (unsigned)d.units * 16 || ((size_t)d.off + d.units) * 16 > L.bytes ||
                    lv_smem(P.end, d.nrows, h->ncols, sizeof(VT)) > L.colour_smem[k])
                    return fail("group larger than its colour's staging buffer");
                const uint32_t *word = (const uint32_t *)(h + 1);
                const uint16_t *rows = (const uint16_t *)(t + P.rows), *place = (const uint16_t *)(t + P.place);
                const int *cols = (const int *)(t + P.cols);
                const VT *dv = (const VT *)(t + P.dinv), *vw = (const VT *)(t + P.val);
                const LvRecord *rec = (const LvRecord *)(t + P.rec);
                const uint16_t *first = (const uint16_t *)(t + P.first);
                if (first[h->steps] != h->nin) return fail("steps do not cover the in-chain slices");
                std::vector<VT> ys;
                std::vector<int> fin(d.nrows, 0);
                for (int i = 0; i < d.nrows; i++) ys.push_back(yy[d.pos0 + i]);
                for (int i = 0; i < h->ncols; i++) {
                    if (cols[i] < 0 || cols[i] >= N || !done[cols[i]]) return fail("gathers a row that is not finished");
                    ys.push_back(yy[cols[i]]);
                }
                ys.push_back(VT(0));
                auto entry = [&](int s, int kk, int lane) { return (size_t)(((word[s] & ~kLvFinal) >> 8) + kk) * 32 + lane; };
                for (int s = 0; s < h->next; s++)
                    for (int q = 0; q < 32; q++) {
                        const unsigned r = rows[s * 32 + q];
                        if (r == kLvNone) continue;
                        if ((int)r >= d.nrows) return fail("row out of the group");
                        VT a = ys[r];
                        for (int kk = 0; kk < (int)(word[s] & 255u); kk++) {
                            const size_t at = entry(s, kk, q);
                            if (at >= (size_t)h->eslots * 32) return fail("entry out of the group's block");
                            const int c = place[at];
                            if (c < d.nrows || c >= (int)ys.size()) return fail("external entry names no gathered row");
                            if (c + 1 == (int)ys.size() && vw[at] != VT(0)) return fail("padding with a value");
                            a -= vw[at] * ys[c];
                            stored += c + 1 < (int)ys.size();
                        }
                        if (word[s] & kLvFinal) a *= dv[r];
                        if (word[s] & kLvFinal) fin[r] = 1;
                        ys[r] = a;
                    }
                const int zero = (int)ys.size() - 1;
                for (int l = 0; l < h->steps; l++) {
                    if (first[l + 1] - first[l] > h->most) return fail("more slices than the header says");
                    std::vector<std::pair<int, VT>> out;  // all slices of a step read before any writes
                    std::vector<int> read(ys.size(), 0);
                    for (int s = first[l]; s < first[l + 1]; s++) {
                        const uint32_t wd = word[h->next + s];
                        const int w = (int)(wd & 255u);
                        if (w < 1 || w > 3) return fail("in-chain slice wider than three");
                        for (int q = 0; q < 32; q++) {
                            const LvRecord &r = rec[s * 32 + q];
                            if (r.row != zero && r.row >= d.nrows) return fail("row out of the group");
                            VT a = ys[r.row];
                            for (int k = 0; k < w; k++) {
                                const size_t at = (size_t)(((wd & ~kLvFinal) >> 8) + k) * 32 + q;
                                if (at >= (size_t)h->slots * 32) return fail("entry out of the group's block");
                                const int c = r.place[3 - w + k];
                                if (c != zero && c >= d.nrows) return fail("in-chain entry outside the group");
                                if (c == zero && vw[at] != VT(0)) return fail("padding with a value");
                                if (c != zero) read[c] = 1;
                                a -= vw[at] * ys[c];
                                stored += c < d.nrows;
                            }
                            if ((wd & kLvFinal) && r.row != zero) a *= dv[r.row];
                            if (r.row != zero) out.push_back({r.row, a});
                            if ((wd & kLvFinal) && r.row != zero) fin[r.row] = 1;
                        }
                    }
                    for (const auto &o : out) {
                        if (read[o.first]) return fail("reads a row of its own step");
                        ys[o.first] = o.second;
                    }
                }
                for (int i = 0; i < d.nrows; i++) {
                    if (upper && !fin[i]) return fail("U row not scaled");
                    next[d.pos0 + i] = ys[i];
                    if (done[d.pos0 + i]) return fail("row in two groups");
                }
            }
            yy = next;
            for (int g = L.colour_groups[k]; g < L.colour_groups[k + 1]; g++)
                for (int i = 0; i < L.groups[g].nrows; i++) done[L.groups[g].pos0 + i] = 1;
        }
        for (int r = 0; r < N; r++) {
            if (!done[r]) return fail("row not in any group");
            y[r] = yy[r];
        }
        if (stored != L.stored) return fail("entries lost");
        return 0;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

}  // namespace

extern "C" int lv_emulate_d(int N, const double *val, const int *cind, const int *rptr, int upper, const int *cptr,
                            int cnum, int bs, int want, int spread, const double *x, double *y, int *info, char *err, int errlen)
{
    return emulate(N, val, cind, rptr, upper, cptr, cnum, bs, want, spread, x, y, info, err, errlen);
}

extern "C" int lv_emulate_s(int N, const float *val, const int *cind, const int *rptr, int upper, const int *cptr,
                            int cnum, int bs, int want, int spread, const float *x, float *y, int *info, char *err, int errlen)
{
    return emulate(N, val, cind, rptr, upper, cptr, cnum, bs, want, spread, x, y, info, err, errlen);
}
