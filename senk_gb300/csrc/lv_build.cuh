// Builds the row-sorted slice layout (lv_layout.hpp) on the device from the
// factor's CSR arrays, in the form and order of make_lv_layout's blocks. On the
// host the layout costs several times what the row slots did (sorting and
// finding the distinct columns of every group); here one CTA builds a group,
// once for its size and once more to write it.
#pragma once

#include "common.cuh"
#include "lv_layout.hpp"

namespace senkgpu {

// One group to build: its rows, and the rows [c0, c1) of its colour.
struct LvJob {
    int pos0, nrows, c0, c1;
};

// What building a group reported.
struct LvSize {
    int units;  // 16-byte units of the block
    int smem;   // bytes of shared memory it needs in k_sweep_lv
    int bad;    // 1: a row does not fit the schedule; 2: larger than this builder's tables
};

constexpr int kLvBuildCols = 4096;    // external entries of a group
constexpr int kLvBuildSlices = 512;
constexpr int kLvBuildOrder = 2 * kLvMaxRows + 32 * 33;  // external and in-chain rows

// Dynamic shared memory of k_lv_build.
struct LvBuildShared {
    int cols[kLvBuildCols];
    uint32_t mask[kLvMaxRows];  // in-chain columns of a row, one bit per chain-local row
    uint32_t word[kLvBuildSlices];
    uint16_t src[kLvBuildSlices], skip[kLvBuildSlices], first[kLvBuildSlices + 2];
    uint16_t ne[kLvMaxRows], ni[kLvMaxRows];
    uint16_t order[kLvBuildOrder];  // rows: external classes, then level after level, each from a multiple of 32 on
    unsigned char lev[kLvMaxRows], cls[kLvMaxRows];
    int count[36], base[36];  // per class: 0, 1 external (final, others), 2.. in-chain levels
    int warp[kLvMaxRows / 32];
    int ncol, nslice, bad;
    LvHeader h;
};

// WRITE = false: sizes only. blockDim = kLvMaxRows.
template <typename VT, bool UPPER, bool WRITE>
__global__ void __launch_bounds__(kLvMaxRows)
k_lv_build(const LvJob *__restrict__ jobs, const VT *__restrict__ val, const int *__restrict__ cind,
           const int *__restrict__ rptr, int n, int bs, const LvGroup *__restrict__ groups, unsigned char *blocks,
           LvSize *size)
{
    extern __shared__ __align__(16) unsigned char lvb[];
    LvBuildShared &S = *reinterpret_cast<LvBuildShared *>(lvb);
    const LvJob d = jobs[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid < 36) S.count[tid] = 0;
    if (tid == 0) {
        S.ncol = 0;
        S.bad = 0;
    }
    for (int i = tid; i < kLvBuildOrder; i += blockDim.x) S.order[i] = (uint16_t)kLvNone;
    __syncthreads();
    // counts and in-chain masks; the checks of make_lv_layout
    const int row = d.pos0 + tid;
    const bool live = tid < d.nrows;
    const int cs = row - row % bs, a = live ? rptr[row] + (UPPER ? 1 : 0) : 0, e = live ? rptr[row + 1] : 0;
    int ne = 0, ni = 0;
    uint32_t mask = 0u;
    if (live) {
        bool ok = !UPPER || (e >= a && cind[a - 1] == row);
        for (int j = a; j < e && ok; j++) {
            const int c = cind[j];
            if (c < 0 || c >= n || (UPPER ? c <= row : c >= row)) ok = false;
            else if (c >= cs && c < cs + bs) {
                ni++;
                mask |= 1u << (c - cs);
            } else if (UPPER ? c < d.c1 : c >= d.c0) ok = false;  // a column of its own or a later colour
            else ne++;
        }
        if (!ok || ne > 255 || ni > 255) S.bad = 1;
    }
    S.ne[tid] = (uint16_t)ne;
    S.ni[tid] = (uint16_t)ni;
    S.mask[tid] = mask;
    S.lev[tid] = 0;
    __syncthreads();
    if (S.bad) {
        if (tid == 0) size[blockIdx.x] = {0, 0, 1};
        return;
    }
    // levels: at most bs rounds
    for (;;) {
        int l = 0;
        for (uint32_t m = mask; m; m &= m - 1) l = max(l, S.lev[cs - d.pos0 + __ffs(m) - 1] + 1);
        const bool change = l != S.lev[tid];
        if (!__syncthreads_or(change)) break;
        S.lev[tid] = (unsigned char)l;
        __syncthreads();
    }
    // classes: external (255: none) and in-chain (level)
    const int lev = S.lev[tid];
    const int ec = !live ? 255 : UPPER && ni == 0 ? 0 : ne > 0 ? 1 : 255;
    S.cls[tid] = (unsigned char)ec;
    if (ec < 2) atomicAdd(&S.count[ec], 1);
    if (live && lev > 0) atomicAdd(&S.count[1 + lev], 1);
    if (ne > 0) {  // the external columns, in any order
        int at = atomicAdd(&S.ncol, ne);
        if (at + ne <= kLvBuildCols)
            for (int j = a; j < e; j++) {
                const int c = cind[j];
                if (c < cs || c >= cs + bs) S.cols[at++] = c;
            }
    }
    __syncthreads();
    const int next_entries = S.ncol;
    if (next_entries > kLvBuildCols) {
        if (tid == 0) size[blockIdx.x] = {0, 0, 2};
        return;
    }
    if (tid == 0) {
        int b = 0;
        for (int k = 0; k < 35; k++) {
            S.base[k] = b;
            b += (S.count[k] + 31) / 32 * 32;
        }
    }
    __syncthreads();
    // a row's place in its class: longest first, ties in row order
    if (ec < 2 || lev > 0) {
        int re = 0, ri = 0;
        for (int q = 0; q < d.nrows; q++) {
            if (S.cls[q] == ec && (S.ne[q] > ne || (S.ne[q] == ne && q < tid))) re++;
            if (S.lev[q] == lev && (S.ni[q] > ni || (S.ni[q] == ni && q < tid))) ri++;
        }
        if (ec < 2) S.order[S.base[ec] + re] = (uint16_t)tid;
        if (live && lev > 0) S.order[S.base[1 + lev] + ri] = (uint16_t)tid;
    }
    // distinct external columns: bitonic sort, then compaction
    int cap = 1;
    while (cap < next_entries) cap *= 2;
    for (int i = next_entries + tid; i < cap; i += blockDim.x) S.cols[i] = INT_MAX;
    __syncthreads();
    for (int k = 2; k <= cap; k *= 2)
        for (int j = k / 2; j > 0; j /= 2) {
            for (int i = tid; i < cap / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (j - 1)), hi = lo + j;
                const int x = S.cols[lo], y = S.cols[hi];
                if ((x > y) == ((lo & k) == 0)) {
                    S.cols[lo] = y;
                    S.cols[hi] = x;
                }
            }
            __syncthreads();
        }
    {
        constexpr int M = kLvBuildCols / kLvMaxRows;
        int mine[M], cnt = 0;
#pragma unroll
        for (int u = 0; u < M; u++) {
            const int i = tid * M + u;
            const bool keep = i < next_entries && (i == 0 || S.cols[i] != S.cols[i - 1]);
            mine[u] = keep ? S.cols[i] : -1;
            cnt += keep;
        }
        int v = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) S.warp[w] = v;
        __syncthreads();
        int before = v - cnt;
        for (int k = 0; k < w; k++) before += S.warp[k];
#pragma unroll
        for (int u = 0; u < M; u++)
            if (mine[u] >= 0) S.cols[before++] = mine[u];
        if (tid == kLvMaxRows - 1) S.ncol = before;
    }
    // slices
    if (tid == 0) {
        LvHeader h{};
        int ns = 0, slots = 0, steps = 0;
        bool fits = true;
        S.first[0] = 0;
        auto add = [&](int src, int wd, int skip, uint32_t flag) {
            if (ns >= kLvBuildSlices || slots > 65535 - 255) {
                fits = false;
                return;
            }
            S.word[ns] = ((uint32_t)slots << 8) | (uint32_t)wd | flag;
            S.src[ns] = (uint16_t)src;
            S.skip[ns] = (uint16_t)skip;
            ns++;
            slots += wd;
        };
        for (int k = 0; k < 2; k++)
            for (int i = 0; i < S.count[k]; i += 32) {
                const int src = S.base[k] + i, wd = S.ne[S.order[src]];
                add(src, wd, wd, k == 0 ? kLvFinal : 0u);
            }
        h.next = (uint16_t)ns;
        h.eslots = (uint16_t)slots;
        for (int l = 1; l < 33 && S.count[1 + l] > 0 && fits; l++) {
            const int base = S.base[1 + l];
            for (int part = (S.ni[S.order[base]] + 2) / 3; part > 0 && fits; part--) {
                const int before = ns;
                for (int i = 0; i < S.count[1 + l] && S.ni[S.order[base + i]] > 3 * (part - 1); i += 32) {
                    const int left = min((int)S.ni[S.order[base + i]], 3 * part);
                    add(base + i, left - 3 * (part - 1), left, UPPER && part == 1 ? kLvFinal : 0u);
                }
                if (!fits || steps + 1 > kLvBuildSlices) {
                    fits = false;
                    break;
                }
                S.first[++steps] = (uint16_t)(ns - h.next);
                h.most = (uint16_t)max((int)h.most, ns - before);
            }
        }
        h.nin = (uint16_t)(ns - h.next);
        h.steps = (uint16_t)steps;
        h.slots = (uint16_t)slots;
        S.h = h;
        S.nslice = ns;
        if (!fits) S.bad = 2;
    }
    __syncthreads();
    if (S.bad) {
        if (tid == 0) size[blockIdx.x] = {0, 0, 2};
        return;
    }
    if (tid == 0) S.h.ncols = (uint16_t)S.ncol;
    __syncthreads();
    const int ncol = S.ncol;
    const LvParts P = lv_parts(S.h, UPPER ? d.nrows * (unsigned)sizeof(VT) : 0u, (unsigned)sizeof(VT));
    if (!WRITE) {
        if (tid == 0) size[blockIdx.x] = {(int)(P.end / 16), (int)lv_smem(P.end, d.nrows, ncol, sizeof(VT)), 0};
        return;
    }
    unsigned char *t = blocks + (size_t)groups[blockIdx.x].off * 16;
    const int ns = S.nslice, steps = S.h.steps;
    for (unsigned i = tid; i < P.place / 4; i += blockDim.x) reinterpret_cast<uint32_t *>(t)[i] = 0u;  // padding
    __syncthreads();
    if (tid == 0) *reinterpret_cast<LvHeader *>(t) = S.h;
    for (int i = tid; i < ns; i += blockDim.x) reinterpret_cast<uint32_t *>(t + sizeof(LvHeader))[i] = S.word[i];
    for (int i = tid; i <= steps; i += blockDim.x) reinterpret_cast<uint16_t *>(t + P.first)[i] = S.first[i];
    for (int i = tid; i < ncol; i += blockDim.x) reinterpret_cast<int *>(t + P.cols)[i] = S.cols[i];
    if (UPPER && live) reinterpret_cast<VT *>(t + P.dinv)[tid] = val[a - 1];
    uint16_t *rows = reinterpret_cast<uint16_t *>(t + P.rows), *place = reinterpret_cast<uint16_t *>(t + P.place);
    LvRecord *rec = reinterpret_cast<LvRecord *>(t + P.rec);
    VT *v = reinterpret_cast<VT *>(t + P.val);
    const int zero = d.nrows + ncol;
    for (int s = w; s < ns; s += kLvMaxRows / 32) {
        const int wd = (int)(S.word[s] & 255u);
        const size_t at = (size_t)((S.word[s] & ~kLvFinal) >> 8) * 32 + lane;
        const bool external = s < S.h.next;
        const unsigned id = S.order[S.src[s] + lane];
        int k = 0;  // columns written
        uint16_t p3[3] = {(uint16_t)zero, (uint16_t)zero, (uint16_t)zero};
        auto put = [&](VT x, int p) {
            v[at + 32 * (size_t)k] = x;
            if (external) place[at + 32 * (size_t)k] = (uint16_t)p;
            else p3[3 - wd + k] = (uint16_t)p;
            k++;
        };
        if (id != kLvNone) {
            const int r = d.pos0 + (int)id, rs = r - r % bs;
            const int b = rptr[r] + (UPPER ? 1 : 0), f = rptr[r + 1];
            int q = (int)S.skip[s] - (external ? S.ne[id] : S.ni[id]);  // column of the row's first entry
            for (; k < wd && k < q;) put(VT(0), zero);
            for (int i = b; i < f && k < wd; i++) {
                const int j = UPPER ? f - 1 - (i - b) : i;
                const int c = cind[j];
                if ((c >= rs && c < rs + bs) == external) continue;
                if (q >= 0) {
                    int p = c - d.pos0;
                    if (external) {  // its place among the distinct columns
                        int lo = 0, hi = ncol - 1;
                        while (lo < hi) {
                            const int m = (lo + hi) / 2;
                            if (S.cols[m] < c) lo = m + 1;
                            else hi = m;
                        }
                        p = d.nrows + lo;
                    }
                    put(val[j], p);
                }
                q++;
            }
        }
        while (k < wd) put(VT(0), zero);
        if (external) {
            rows[s * 32 + lane] = (uint16_t)id;
        } else {
            LvRecord r;
            r.row = (uint16_t)(id == kLvNone ? (unsigned)zero : id);
            r.place[0] = p3[0];
            r.place[1] = p3[1];
            r.place[2] = p3[2];
            rec[(s - S.h.next) * 32 + lane] = r;
        }
    }
}

}  // namespace senkgpu
