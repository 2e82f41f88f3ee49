// Row-sorted slice layout of a triangular factor for the colour sweeps
// (k_sweep_lv in kernels.cuh). Host-only code: it builds plain arrays that the
// plan uploads, and a CPU emulation of the kernel can build them too.
//
// The schedule is a list of colours (row ranges, in processing order); a chain
// is `bs` consecutive rows of one colour, solved in order. A group is up to
// 512 consecutive rows of one colour (whole chains). Its entries come in
// slices of 32 rows, slot-major: entry k of the slice's row `lane` is element
// (slice slot + k) * 32 + lane, the slice as wide as its longest row.
//  * External slices hold the entries whose columns lie outside the row's
//    chain (rows of earlier colours), the group's rows taken longest first.
//  * In-chain slices hold the entries inside the chain, by dependency level:
//    a row is at level 1 + the largest level of the rows of its chain it reads
//    (0: it reads none and has no in-chain slice). Rows of one level, over all
//    chains of the group, are independent; longest first. A slice is at most
//    three wide and a step holds slices of different rows only: a level with
//    longer rows takes several steps, the last one of three entries.
// So a warp's 32 lanes have (nearly) equal work in both parts, and a chain
// costs as many steps as its rows depend on one another (about five for the 16
// rows of a breadth-first block of a 7-point grid), not one per row. Each row's
// entries keep the reference's subtraction order (include/senk_sparse.hpp:
// 250-315: ascending columns for L, descending for U, external ones first).
//
// The group lists the distinct external columns it reads, ascending; the
// kernel gathers each once, neighbouring lanes from neighbouring rows, and an
// entry names its operand by a 16-bit place: a row of the group (< nrows, an
// in-chain column), nrows + j (the j-th external column), or the place after
// the last (a zero; padding, with value 0).
//
// Block of a group, from 16-byte unit `off`, each part padded to 16 bytes:
// LvHeader; one word per slice (slot << 8 | width; external slices first, then
// step after step); the in-chain slices before each step (steps + 1 numbers of
// 16 bits; kLvFinal in a word, U only: the slice finishes its rows, so
// it multiplies them by their inverted diagonal; external slices of rows
// without in-chain entries are kept apart for that); 32 row numbers of 16 bits
// per external slice (group row; kLvNone: no row); 32 records of 8 bytes per
// in-chain slice ({row, three places}, the last `width` places in use); the
// external columns; U: the rows' inverted diagonal; the external entries'
// places; all entries' values.
#pragma once

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

namespace senkgpu {

struct LvGroup {
    int pos0;   // first row
    int nrows;  // rows (<= 512)
    int off;    // block: first 16-byte unit
    int units;  // and 16-byte units
};
static_assert(sizeof(LvGroup) == 16, "LvGroup is one 16-byte load");

constexpr int kLvMaxRows = 512;
constexpr unsigned kLvNone = 0xffffu;
constexpr uint32_t kLvFinal = 0x80000000u;

struct LvHeader {
    uint16_t next;    // external slices
    uint16_t nin;     // in-chain slices
    uint16_t steps;   // in-chain steps
    uint16_t most;    // slices of the step that has most
    uint16_t ncols;   // external columns
    uint16_t eslots;  // 32-entry slots of the external slices
    uint16_t slots;   // and of all slices
    uint16_t pad;
};
static_assert(sizeof(LvHeader) == 16, "the slice words follow at byte 16");

struct LvRecord {
    uint16_t row, place[3];
};
static_assert(sizeof(LvRecord) == 8, "LvRecord is one 8-byte load");

// Byte offsets of a group's block.
struct LvParts {
    unsigned first, rows, rec, cols, dinv, place, val, end;
};
#ifndef SENK_HD
#ifdef __CUDACC__
#define SENK_HD __host__ __device__
#else
#define SENK_HD
#endif
#endif
SENK_HD constexpr unsigned lv_round(unsigned b) { return (b + 15u) / 16u * 16u; }
SENK_HD constexpr LvParts lv_parts(const LvHeader &h, unsigned dinv_bytes, unsigned vb)
{
    LvParts p{};
    p.first = 16u + 4u * ((unsigned)h.next + h.nin);
    p.rows = lv_round(p.first + 2u * (h.steps + 1u));
    p.rec = p.rows + 64u * h.next;
    p.cols = p.rec + 256u * h.nin;
    p.dinv = p.cols + lv_round(4u * h.ncols);
    p.place = p.dinv + lv_round(dinv_bytes);
    p.val = p.place + 64u * h.eslots;
    p.end = p.val + 32u * vb * h.slots;
    return p;
}

// Shared memory a group needs: its block, then its operands (rows, external
// columns, the zero).
constexpr size_t lv_smem(size_t block, size_t nrows, size_t cols, size_t vb) { return block + (nrows + cols + 1) * vb; }

template <typename VT>
struct LvLayout {
    std::vector<LvGroup> groups;  // in processing order
    std::unique_ptr<unsigned char[]> blocks;
    size_t bytes = 0;
    std::vector<int> colour_groups;
    std::vector<size_t> colour_smem;  // most shared memory of a group of each colour
    std::vector<int> colour_rows;     // rows per group of each colour
    long long stored = 0;
};

// Distinct columns of a group, ascending, and the place of each: a hash table
// of aligned runs of 32 columns, each with a bit per column.
class LvColumns {
    struct Run {
        int key;
        uint32_t bits;
        int before;  // distinct columns of smaller runs
    };
    std::vector<Run> slot;
    std::vector<int> used;
    unsigned mask = 0;
    Run &find(int key)
    {
        unsigned i = ((unsigned)key * 2654435761u) & mask;
        while (slot[i].key >= 0 && slot[i].key != key) i = (i + 1) & mask;
        return slot[i];
    }

public:
    // room for `n` columns
    void reset(size_t n)
    {
        size_t cap = 64;
        while (cap < 2 * n) cap *= 2;
        if (cap > slot.size()) slot.assign(cap, Run{-1, 0u, 0});
        else
            for (int i : used) slot[i] = Run{-1, 0u, 0};
        used.clear();
        mask = (unsigned)slot.size() - 1;
    }
    void add(int c)
    {
        Run &r = find(c >> 5);
        if (r.key < 0) {
            r.key = c >> 5;
            used.push_back((int)(&r - slot.data()));
        }
        r.bits |= 1u << (c & 31);
    }
    void finish(std::vector<int> &cols)
    {
        std::sort(used.begin(), used.end(), [&](int a, int b) { return slot[a].key < slot[b].key; });
        cols.clear();
        for (int i : used) {
            slot[i].before = (int)cols.size();
            for (uint32_t m = slot[i].bits; m; m &= m - 1) cols.push_back(slot[i].key * 32 + __builtin_ctz(m));
        }
    }
    int place(int c)
    {
        const Run &r = find(c >> 5);
        return r.before + __builtin_popcount(r.bits & ((1u << (c & 31)) - 1u));
    }
};

// `rows` in order of descending cnt, ties in row order.
inline void lv_sort(std::vector<int> &rows, std::vector<int> &tmp, const unsigned char *cnt)
{
    int start[257] = {};
    for (int r : rows) start[255 - cnt[r] + 1]++;
    for (int k = 0; k < 256; k++) start[k + 1] += start[k];
    tmp.resize(rows.size());
    for (int r : rows) tmp[start[255 - cnt[r]]++] = r;
    rows.swap(tmp);
}

// The groups (rows only) of each colour: 512 rows each, halved while some
// group's entries take more than `want` bytes (down to one chain or 32 rows) or
// the colour has fewer than `spread` groups (down to 64 rows).
inline void lv_cut(std::vector<LvGroup> &gd, std::vector<int> &colour_groups, std::vector<int> &colour_rows,
                   const int *rptr, const std::vector<std::pair<int, int>> &colours, int bs, size_t want, int spread,
                   size_t vb)
{
    gd.clear();
    colour_groups.assign(1, 0);
    colour_rows.clear();
    for (const auto &c : colours) {
        int gr = kLvMaxRows;
        for (;; gr /= 2) {
            size_t worst = 0;
            for (int p = c.first; p < c.second; p += gr)
                worst = std::max(worst, (size_t)(rptr[std::min(p + gr, c.second)] - rptr[p]) * (2 + vb));
            const bool more = worst > want || (gr > 64 && (long long)gr * spread > c.second - c.first);
            if (!more || gr / 2 < std::max(32, bs)) break;
        }
        for (int p = c.first; p < c.second; p += gr) gd.push_back({p, std::min(gr, c.second - p), 0, 0});
        colour_groups.push_back((int)gd.size());
        colour_rows.push_back(gr);
    }
}

// Builds the layout of one factor. colour_of[row]: the colour's index in
// processing order; `want` and `spread` as for lv_cut.
// Throws std::invalid_argument when the factor does not fit the schedule;
// returns false when a group's block would need more than `most` bytes.
template <typename VT>
bool make_lv_layout(LvLayout<VT> &out, bool upper, int N, const VT *val, const int *cind, const int *rptr,
                    const std::vector<std::pair<int, int>> &colours, int bs, const int *colour_of, size_t want,
                    int spread, size_t most)
{
    if (bs < 1 || bs > 32 || N % bs) throw std::invalid_argument("chain length must divide N and be at most 32");
    std::vector<unsigned char> ne(N), ni(N), lev(N);
    int bad = -1;
    long long stored = 0;
#pragma omp parallel for schedule(static) reduction(+ : stored)
    for (int b = 0; b < N / bs; b++) {
        const int cs = b * bs, ce = cs + bs;
        bool ok = true;
        for (int st = 0; st < bs && ok; st++) {
            const int row = upper ? ce - 1 - st : cs + st;  // solve order
            const int j0 = rptr[row] + (upper ? 1 : 0), j1 = rptr[row + 1];
            if (upper) ok = j1 >= j0 && cind[j0 - 1] == row;  // a U row starts with its diagonal
            int re = 0, ri = 0, l = 0;
            for (int j = j0; j < j1 && ok; j++) {
                const int c = cind[j];
                if (c < 0 || c >= N || (upper ? c <= row : c >= row)) ok = false;
                else if (c >= cs && c < ce) {
                    ri++;
                    l = std::max(l, lev[c] + 1);
                } else if (colour_of[c] >= colour_of[row]) ok = false;  // must be final before this colour
                else re++;
            }
            ok = ok && re <= 255 && ri <= 255;
            ne[row] = (unsigned char)re;
            ni[row] = (unsigned char)ri;
            lev[row] = (unsigned char)l;
            stored += re + ri;
        }
        if (!ok) {
#pragma omp atomic write
            bad = b;
        }
    }
    if (bad >= 0)
        throw std::invalid_argument(std::string(upper ? "U" : "L") + " factor rows of chain " + std::to_string(bad) +
                                    " do not fit the schedule (diagonal first in U, strictly triangular, columns of "
                                    "other chains in earlier colours, at most 255 entries)");
    long long covered = 0;
    for (const auto &c : colours) {
        if (c.first % bs || c.second % bs || c.second < c.first || c.first < 0 || c.second > N)
            throw std::invalid_argument("colour range not made of whole chains");
        covered += c.second - c.first;
    }
    if (covered != N) throw std::invalid_argument("colours do not cover the N rows");
    std::vector<LvGroup> gd;
    lv_cut(gd, out.colour_groups, out.colour_rows, rptr, colours, bs, want, spread, sizeof(VT));
    const int ng = (int)gd.size();
    std::vector<std::vector<unsigned char>> block(ng);
    std::vector<size_t> smem(ng);
    bool wide = false;
#pragma omp parallel reduction(|| : wide)
    {
        LvColumns table;
        std::vector<uint32_t> word;
        std::vector<uint16_t> srow, first, skip;  // 32 rows per slice; see add()
        std::vector<int> cols, rows, tmp;
        std::vector<uint16_t> pl(256);
#pragma omp for schedule(dynamic, 16)
        for (int g = 0; g < ng; g++) {
            const int p0 = gd[g].pos0, nrows = gd[g].nrows;
            const unsigned char *gne = ne.data() + p0, *gni = ni.data() + p0, *glev = lev.data() + p0;
            LvHeader h{};
            word.clear();
            srow.clear();
            skip.clear();
            rows.clear();
            first.assign(1, 0);
            size_t slots = 0;
            // a slice of rows[i..i+32), `w` wide, that starts `from_end` entries
            // before its rows' last
            auto add = [&](size_t i, int w, int from_end, uint32_t flag) {
                word.push_back(((uint32_t)slots << 8) | (uint32_t)w | flag);
                skip.push_back((uint16_t)from_end);
                for (size_t q = i; q < i + 32; q++) srow.push_back((uint16_t)(q < rows.size() ? (unsigned)rows[q] : kLvNone));
                slots += w;
            };
            auto add_external = [&](uint32_t flag) {
                lv_sort(rows, tmp, gne);
                for (size_t i = 0; i < rows.size(); i += 32) add(i, gne[rows[i]], gne[rows[i]], flag);
                rows.clear();
            };
            // external part: U's rows without in-chain entries (finished here,
            // so those without any entry too), then the rows with external entries
            if (upper) {
                for (int r = 0; r < nrows; r++)
                    if (!gni[r]) rows.push_back(r);
                add_external(kLvFinal);
            }
            for (int r = 0; r < nrows; r++)
                if (gne[r] && (gni[r] || !upper)) rows.push_back(r);
            add_external(0u);
            h.next = (uint16_t)word.size();
            h.eslots = (uint16_t)slots;
            const size_t eslots = slots;
            int nlev = 0;
            for (int r = 0; r < nrows; r++) nlev = std::max<int>(nlev, glev[r]);
            for (int d = 1; d <= nlev; d++) {
                for (int r = 0; r < nrows; r++)
                    if (glev[r] == d) rows.push_back(r);
                lv_sort(rows, tmp, gni);
                for (int part = (gni[rows[0]] + 2) / 3; part > 0; part--) {
                    // the slices with at least `part` steps left; the last
                    // `part` steps of a slice take its entries three at a time
                    for (size_t i = 0; i < rows.size() && gni[rows[i]] > 3 * (part - 1); i += 32) {
                        const int left = std::min<int>(gni[rows[i]], 3 * part);
                        add(i, left - 3 * (part - 1), left, upper && part == 1 ? kLvFinal : 0u);
                    }
                    first.push_back((uint16_t)(word.size() - h.next));
                    h.most = std::max<uint16_t>(h.most, (uint16_t)(first.back() - first[first.size() - 2]));
                }
                rows.clear();
            }
            // the external columns
            size_t ext = 0;
            for (int r = 0; r < nrows; r++) ext += gne[r];
            table.reset(ext);
            for (int row = p0; row < p0 + nrows; row++)
                for (int j = rptr[row] + (upper ? 1 : 0), cs = row - row % bs; j < rptr[row + 1]; j++)
                    if (cind[j] < cs || cind[j] >= cs + bs) table.add(cind[j]);
            table.finish(cols);
            const size_t steps = first.size() - 1;
            if (slots > 65535 || word.size() > 65535 || cols.size() + nrows >= 65535) {
                wide = true;
                continue;
            }
            h.nin = (uint16_t)(word.size() - h.next);
            h.steps = (uint16_t)steps;
            h.ncols = (uint16_t)cols.size();
            h.eslots = (uint16_t)eslots;
            h.slots = (uint16_t)slots;
            const LvParts P = lv_parts(h, upper ? (unsigned)(nrows * sizeof(VT)) : 0u, (unsigned)sizeof(VT));
            block[g].resize(P.end);
            gd[g].units = (int)(P.end / 16);
            smem[g] = lv_smem(P.end, nrows, cols.size(), sizeof(VT));
            unsigned char *t = block[g].data();
            std::memcpy(t, &h, sizeof(LvHeader));
            if (!word.empty()) std::memcpy(t + sizeof(LvHeader), word.data(), 4 * word.size());
            std::memcpy(t + P.first, first.data(), 2 * first.size());
            if (h.next) std::memcpy(t + P.rows, srow.data(), 64 * (size_t)h.next);
            if (!cols.empty()) std::memcpy(t + P.cols, cols.data(), 4 * cols.size());
            if (upper)
                for (int r = 0; r < nrows; r++)
                    std::memcpy(t + P.dinv + r * sizeof(VT), &val[rptr[p0 + r]], sizeof(VT));
            uint16_t *place = reinterpret_cast<uint16_t *>(t + P.place);
            LvRecord *rec = reinterpret_cast<LvRecord *>(t + P.rec);
            VT *v = reinterpret_cast<VT *>(t + P.val);
            const uint16_t zero = (uint16_t)(nrows + (int)cols.size());
            for (size_t s = 0; s < word.size(); s++) {
                const int w = (int)(word[s] & 255u);
                const bool external = s < h.next;
                for (int q = 0; q < 32; q++) {
                    const size_t at = (size_t)((word[s] & ~kLvFinal) >> 8) * 32 + q;
                    const unsigned id = srow[s * 32 + q];
                    for (int k = 0; k < w; k++) {  // padding unless an entry follows
                        v[at + 32 * (size_t)k] = VT(0);
                        pl[k] = zero;
                    }
                    if (id != kLvNone) {
                        const int row = p0 + (int)id;
                        const int cs = row - row % bs, ce = cs + bs;
                        const int a = rptr[row] + (upper ? 1 : 0), e = rptr[row + 1];
                        int k = (int)skip[s] - (external ? gne[id] : gni[id]);
                        for (int i = a; i < e; i++) {
                            const int j = upper ? e - 1 - (i - a) : i;
                            const int c = cind[j];
                            const bool in = c >= cs && c < ce;
                            if (in == external) continue;
                            if (k >= 0 && k < w) {
                                v[at + 32 * (size_t)k] = val[j];
                                pl[k] = (uint16_t)(in ? c - p0 : nrows + table.place(c));
                            }
                            k++;
                        }
                    }
                    if (external) {
                        for (int k = 0; k < w; k++) place[at + 32 * (size_t)k] = pl[k];
                    } else {
                        LvRecord &r = rec[(s - h.next) * 32 + q];
                        r.row = (uint16_t)(id == kLvNone ? zero : id);
                        for (int k = 0; k < 3; k++) r.place[k] = k < 3 - w ? zero : pl[k - (3 - w)];
                    }
                }
            }
        }
    }
    if (wide) return false;
    long long units = 0;
    for (int g = 0; g < ng; g++) {
        gd[g].off = (int)units;
        units += gd[g].units;
        if (units >= INT_MAX) throw std::invalid_argument("factor too large for 32-bit block offsets");
        if (smem[g] > most) return false;
    }
    out.colour_smem.assign(colours.size(), 0);
    for (size_t c = 0; c < colours.size(); c++)
        for (int g = out.colour_groups[c]; g < out.colour_groups[c + 1]; g++)
            out.colour_smem[c] = std::max(out.colour_smem[c], smem[g]);
    out.bytes = (size_t)std::max<long long>(units, 1) * 16;
    out.blocks.reset(new unsigned char[out.bytes]);
#pragma omp parallel for schedule(dynamic, 64)
    for (int g = 0; g < ng; g++) {
        std::memcpy(out.blocks.get() + (size_t)gd[g].off * 16, block[g].data(), block[g].size());
        std::vector<unsigned char>().swap(block[g]);
    }
    out.groups = std::move(gd);
    out.stored = stored;
    return true;
}

}  // namespace senkgpu
