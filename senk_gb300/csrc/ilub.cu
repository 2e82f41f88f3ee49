// ILUB: triangular sweeps on BCSR factors (include/senk_sparse.hpp:392-465
// sequential, 481-581 ABMC).
//
// Semantics kept from the reference, block row by block row (i = first row):
//  L: y[i..i+bnl) = x; for every block in ascending order and every column l of
//     it, all rows of the block row subtract bval * y[col]. The reference's row
//     loop is `omp simd`, built by g++ -O3 from vectors of two doubles: y[col]
//     is read again for each pair of rows (r, r+1), after the pairs before it
//     were updated. That is visible when a block holds a value on the diagonal:
//     Csr2Bcsr (include/senk_matrix.hpp:144-211) gives an empty L row the first
//     entry of the next row, so the first row of every block row without lower
//     entries carries one. Rows in a later pair than row `col` see its updated
//     value, rows in its own or an earlier pair the value before the step.
//  U: y[i..i+bnl) = x; the blocks right of the diagonal square in descending
//     order (their columns ascending within a block) as above; then the
//     bnl/bnw diagonal blocks column by column from the right: y[idx] *=
//     (inverted diagonal), then every row above subtracts bval * y[idx].
// One group of G lanes (G = bnl rounded up to a power of two) sweeps one chain;
// lane k holds row i+k. A column inside the block row is read from its lane by
// a shuffle before the step's update; any other column is final in global
// memory (an earlier phase, or an earlier block row of the same chain, written
// by this group before its __syncwarp).
#include <algorithm>
#include <vector>

#include "device.hpp"

namespace senkgpu {

namespace {

template <int BNL>
constexpr int group_lanes()
{
    return BNL <= 1 ? 1 : BNL <= 2 ? 2 : BNL <= 4 ? 4 : BNL <= 8 ? 8 : BNL <= 16 ? 16 : 32;
}

template <typename T, int BNL, int BNW, bool UPPER>
__global__ void __launch_bounds__(kThreads)
k_ilub_sweep(const T *__restrict__ bval, const int *__restrict__ bcind, const int *__restrict__ brptr,
             const int2 *__restrict__ chains, int nch, const T *x, T *y, const int *gate)
{
    if (gated(gate)) return;
    constexpr int G = group_lanes<BNL>();
    constexpr int BS = BNL * BNW;
    constexpr int BREM = BNL / BNW;
    const int lane = threadIdx.x % G;
    const int gid = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) / G);
    if (gid >= nch) return;  // uniform over the group
    const unsigned mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (((threadIdx.x & 31) / G) * G));
    const int2 ch = chains[gid];
    for (int q = 0; q < ch.y; q++) {
        const int br = UPPER ? ch.x + ch.y - 1 - q : ch.x + q;
        const int i = br * BNL;
        T t = lane < BNL ? x[i + lane] : T(0);
        const int b0 = brptr[br], b1 = brptr[br + 1];
        // Blocks are taken kBatch at a time: their columns, values and (for
        // columns outside this block row) y entries are all loaded before the
        // first subtraction, which then run in the blocks' order as before.
        constexpr int kBatch = 4;
        if (!UPPER) {
            for (int j0 = b0; j0 < b1; j0 += kBatch) {
                int xb[kBatch];
                T vv[kBatch][BNW], yy[kBatch][BNW];
#pragma unroll
                for (int u = 0; u < kBatch; u++) xb[u] = j0 + u < b1 ? bcind[j0 + u] * BNW : i;
#pragma unroll
                for (int u = 0; u < kBatch; u++)
#pragma unroll
                    for (int l = 0; l < BNW; l++) {
                        const int rel = xb[u] + l - i;
                        const bool live = j0 + u < b1;
                        vv[u][l] = live && lane < BNL ? bval[(size_t)(j0 + u) * BS + l * BNL + lane] : T(0);
                        yy[u][l] = live && !(rel >= 0 && rel < BNL) ? y[xb[u] + l] : T(0);
                    }
#pragma unroll
                for (int u = 0; u < kBatch; u++) {
                    if (j0 + u >= b1) break;
#pragma unroll
                    for (int l = 0; l < BNW; l++) {
                        const int rel = xb[u] + l - i;
                        const T v = vv[u][l];
                        if (rel >= 0 && rel < BNL) {
                            const T s0 = __shfl_sync(mask, t, rel, G);
                            const T t0 = t - v * s0;
                            const T s1 = __shfl_sync(mask, t0, rel, G);  // y[col] after its own pair
                            t = (lane >> 1) > (rel >> 1) ? t - v * s1 : t0;
                        } else {
                            t -= v * yy[u][l];
                        }
                    }
                }
            }
        } else {
            // blocks right of the diagonal square, from the last one down
            for (int j0 = b1 - 1; j0 >= b0 + BREM; j0 -= kBatch) {
                T vv[kBatch][BNW], yy[kBatch][BNW];
#pragma unroll
                for (int u = 0; u < kBatch; u++) {
                    const int j = j0 - u;
                    const bool live = j >= b0 + BREM;
                    const int xb = live ? bcind[j] * BNW : 0;
#pragma unroll
                    for (int l = 0; l < BNW; l++) {
                        vv[u][l] = live && lane < BNL ? bval[(size_t)j * BS + l * BNL + lane] : T(0);
                        yy[u][l] = live ? y[xb + l] : T(0);
                    }
                }
#pragma unroll
                for (int u = 0; u < kBatch; u++) {
                    if (j0 - u < b0 + BREM) break;
#pragma unroll
                    for (int l = 0; l < BNW; l++) t -= vv[u][l] * yy[u][l];
                }
            }
#pragma unroll
            for (int m = BREM - 1; m >= 0; m--) {
                const T *blk = bval + (size_t)(b0 + m) * BS;
#pragma unroll
                for (int jj = BNW - 1; jj >= 0; jj--) {
                    const int idx = m * BNW + jj;
                    if (lane == idx) t *= blk[jj * BNL + idx];
                    const T s = __shfl_sync(mask, t, idx, G);
                    if (lane < idx) t -= blk[jj * BNL + lane] * s;
                }
            }
        }
        if (lane < BNL) y[i + lane] = t;
        __syncwarp(mask);
    }
}


// ------------------------------------------------ ABMC: slices of block rows
// Chains of one colour, RPW = 32 / BNL (rounded down) to a group: lane
// g * BNL + r holds row r of chain g's block row in every phase, and step q of
// a group is the q-th block row of its chains. A block row's blocks outside its
// chain (rows of earlier colours, which come first in the reference's order)
// are its external slots, the others its in-chain slots; a step is as wide as
// its widest block row (padding: column -1, value 0).
struct BlGroup {
    int row0;  // first block row
    int nch;   // chains
    int ext;   // first external slot (BNW * 32 values each)
    int blob;  // first 16-byte unit of the staged part
};

constexpr int kBlMaxSteps = 16;
constexpr size_t kBlMaxSmem = 160 * 1024;  // shared memory of a group; the kernels' limit for every plan

// Byte offsets of a group's staged part: widths (external, in-chain) of each
// step, the external block columns, the in-chain columns (scalar, from the
// chain's first row), the in-chain values and U's diagonal squares.
struct BlParts {
    unsigned cols, lc, val, diag, end;
};
__host__ __device__ inline BlParts bl_parts(int per, int we, int wi, int rpw, int bnl, int bnw, bool upper, unsigned vb)
{
    auto up = [](unsigned b) { return (b + 15u) / 16u * 16u; };
    BlParts p;
    p.cols = up(4u * per);
    p.lc = p.cols + up(4u * we * rpw);
    p.val = p.lc + up(4u * wi * rpw);
    p.diag = p.val + 32u * vb * wi * bnw;
    p.end = p.diag + (upper ? 32u * vb * per * bnl : 0u);
    return p;
}

// Fills a group's external values and staged part from the BCSR factor. One
// CTA per group, warp q = step q.
template <typename T, int BNL, int BNW, bool UPPER>
__global__ void __launch_bounds__(32 * kBlMaxSteps)
k_ilub_fill(const BlGroup *__restrict__ groups, const uint16_t *__restrict__ widths, int per, int nbr,
            const T *__restrict__ bval, const int *__restrict__ bcind, const int *__restrict__ brptr, T *ext,
            unsigned char *blob)
{
    constexpr int RPW = 32 / BNL, BS = BNL * BNW, BREM = BNL / BNW;
    const BlGroup d = groups[blockIdx.x];
    const uint16_t *wd = widths + (size_t)blockIdx.x * 2 * per;
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / BNL, r = lane % BNL;
    int we0 = 0, wi0 = 0, we = 0, wi = 0;
    for (int k = 0; k < per; k++) {
        if (k == q) {
            we0 = we;
            wi0 = wi;
        }
        we += wd[k];
        wi += wd[per + k];
    }
    const BlParts P = bl_parts(per, we, wi, RPW, BNL, BNW, UPPER, sizeof(T));
    unsigned char *t = blob + (size_t)d.blob * 16;
    if (lane == 0) {
        reinterpret_cast<uint16_t *>(t)[q] = wd[q];
        reinterpret_cast<uint16_t *>(t)[per + q] = wd[per + q];
    }
    int *cols = reinterpret_cast<int *>(t + P.cols), *lc = reinterpret_cast<int *>(t + P.lc);
    T *val = reinterpret_cast<T *>(t + P.val), *diag = reinterpret_cast<T *>(t + P.diag);
    T *xv = ext + (size_t)d.ext * BNW * 32;
    const int br = d.row0 + g * per + q, first = (d.row0 + g * per) * BNL, last = first + per * BNL;
    const bool live = g < RPW && g < d.nch && br < nbr;
    int ke = 0, ki = 0;
    if (live) {
        const int a = brptr[br] + (UPPER ? BREM : 0), e = brptr[br + 1];
        for (int i = a; i < e; i++) {
            const int j = UPPER ? e - 1 - (i - a) : i;
            const int c = bcind[j] * BNW;
            const bool in = c >= first && c < last;
            T *to = in ? val + (size_t)(wi0 + ki) * BNW * 32 : xv + (size_t)(we0 + ke) * BNW * 32;
            for (int l = 0; l < BNW; l++) to[l * 32 + lane] = bval[(size_t)j * BS + l * BNL + r];
            if (r == 0) {
                if (in) lc[(wi0 + ki) * RPW + g] = c - first;
                else cols[(we0 + ke) * RPW + g] = bcind[j];
            }
            if (in) ki++;
            else ke++;
        }
    }
    for (; ke < wd[q]; ke++) {
        for (int l = 0; l < BNW; l++) xv[((size_t)(we0 + ke) * BNW + l) * 32 + lane] = T(0);
        if (r == 0 && g < RPW) cols[(we0 + ke) * RPW + g] = -1;
    }
    for (; ki < wd[per + q]; ki++) {
        for (int l = 0; l < BNW; l++) val[((size_t)(wi0 + ki) * BNW + l) * 32 + lane] = T(0);
        if (r == 0 && g < RPW) lc[(wi0 + ki) * RPW + g] = -1;
    }
    if (UPPER)
        for (int c = 0; c < BNL; c++)  // column c of the diagonal square
            diag[((size_t)q * BNL + c) * 32 + lane] =
                live ? bval[(size_t)(brptr[br] + c / BNW) * BS + (c % BNW) * BNL + r] : T(0);
}

// t -= v[k][l] * gy[k][l] over the last n of B slots, in order (n the same in
// the whole warp); the entry is a jump, see sub_last.
template <int BNW, int B, typename T>
__device__ __forceinline__ void sub_slots(T &t, const T (&v)[B][BNW], const T *gy, int stride, int n)
{
    auto slot = [&](int k) {
#pragma unroll
        for (int l = 0; l < BNW; l++) t -= v[k][l] * gy[k * stride + l];
    };
    switch (n) {
    case 4: if constexpr (B >= 4) slot(B - 4);
    case 3: if constexpr (B >= 3) slot(B - 3);
    case 2: slot(B - 2);
    case 1: slot(B - 1);
    default: break;
    }
}

// One colour per launch, one CTA per group: the block rows of earlier colours
// that the group's external slots name are gathered into shared memory, warp q
// subtracts the external slots of step q (their values read straight into
// registers, a batch of slots ahead), and one warp runs the in-chain part step by
// step, as k_ilub_sweep does. The staged part (TMA) and the first external values
// are read before the wait on the previous kernel, from the third colour on
// (order 2; 0 and 1: the first and the second) x and the gate too. The first
// colour lets the next one start at once, the others after their own wait, so
// whatever wrote x before the sweep, another plan's sweep included, has completed
// when the second colour passes its wait. (k_sweep_lv lets every next colour
// start after its wait and reads x early from the second on; here the colours'
// CTAs, 2.3 to an SM, then fall up to 5 to an SM instead of 4, 175 us instead of
// 152.) Same operations in the same order as k_ilub_sweep, which walked a chain's
// block rows one after another with a dependent gather per four blocks.
// Block-3x3 system, 48^3 nodes (8 colours), one application: FP64 0.524 ->
// 0.151 ms, FP32 0.100 ms. It is bound by a colour's dependent steps (a block
// row's up to 69 FP64 subtractions at 65 cycles, then four in-chain steps) and
// by the FP64 unit (50 us of the 151). FP64 takes two slots ahead in 64
// registers: more CTAs on an SM hide those steps better than four slots in 80
// do (48^3 0.177 ms, 80^3 0.446 against 0.430, 96^3 0.778 against 0.720; 64^3
// 0.238 against 0.246).
template <typename T> constexpr int bl_batch = sizeof(T) == 8 ? 2 : 4;
template <typename T> constexpr int bl_min_blocks = sizeof(T) == 8 ? 4 : 0;  // 0: not stated
template <typename T, int BNL, int BNW, bool UPPER>
__global__ void __launch_bounds__(256, bl_min_blocks<T>)
k_ilub_slices(const BlGroup *__restrict__ groups, int g0, int per, int n, const T *__restrict__ ext,
              const uint4 *__restrict__ blob, const T *x, T *y, const int *gate, int *status, int order)
{
    const bool early_x = order >= 2;
    constexpr int RPW = 32 / BNL, B = bl_batch<T>;
    extern __shared__ __align__(128) unsigned char bls[];
    __shared__ __align__(8) unsigned long long bar;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, nt = blockDim.x, nw = nt >> 5;
    const int g = lane / BNL, r = lane % BNL;
    const BlGroup d = groups[g0 + blockIdx.x], d1 = groups[g0 + blockIdx.x + 1];
    const unsigned bytes = (unsigned)(d1.blob - d.blob) * 16u;
    const int we = d1.ext - d.ext;  // external slots
    const int r0 = d.row0 * BNL, nrows = min(d.nch * per * BNL, n - r0);
    T *ysh = reinterpret_cast<T *>(bls + bytes);  // the group's rows
    T *gy = ysh + RPW * kBlMaxSteps * BNL;        // external operands, slot after slot
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, bytes);
        bulk_g2s(bls, blob + d.blob, bytes, &bar);
    }
    bool skip = false;
    if (early_x) {
        for (int i = tid; i < nrows; i += nt) ysh[i] = x[r0 + i];
        skip = gated(gate);
    }
    if (order == 0) pdl_launch_dependents();
    __syncthreads();
    const bool ok = mbar_wait_bounded(&bar, 0, kWaitLimit);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) atomicExch(status, 2);
        if (!ok) mbar_wait_bounded(&bar, 0, kWaitLimit);
        pdl_wait();
        return;
    }
    const uint16_t *wd = reinterpret_cast<const uint16_t *>(bls);
    int wi = 0, s0 = 0;  // in-chain slots; external slots before step w
    for (int k = 0; k < per; k++) {
        wi += wd[per + k];
        if (k < w) s0 += wd[k];
    }
    const BlParts P = bl_parts(per, we, wi, RPW, BNL, BNW, UPPER, sizeof(T));
    const int *cols = reinterpret_cast<const int *>(bls + P.cols);
    const int *lc = reinterpret_cast<const int *>(bls + P.lc);
    const T *val = reinterpret_cast<const T *>(bls + P.val), *diag = reinterpret_cast<const T *>(bls + P.diag);
    // external values of step q: up to B slots ending at slot k1 of the step
    T v[B][BNW];
    auto load = [&](int first, int k1) {
#pragma unroll
        for (int u = 0; u < B; u++)
            if (k1 - B + u >= 0)
#pragma unroll
                for (int l = 0; l < BNW; l++)
                    v[u][l] = ld_stream(ext + ((size_t)(d.ext + first + k1 - B + u) * BNW + l) * 32 + lane);
    };
    int q = w, width = q < per ? wd[q] : 0, k1 = width > 0 ? (width - 1) % B + 1 : 0;
    if (k1 > 0) load(s0, k1);
    pdl_wait();  // the previous colour (or the producer of x) has finished
    if (order > 0) pdl_launch_dependents();
    if (!early_x) {
        skip = gated(gate);
        for (int i = tid; i < nrows; i += nt) ysh[i] = x[r0 + i];
    }
    if (skip) return;
    for (int i = tid; i < we * RPW * BNW; i += 4 * nt) {
        T a[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int at = i + u * nt, c = at < we * RPW * BNW ? cols[at / BNW] : -1;
            a[u] = c >= 0 ? y[c * BNW + at % BNW] : T(0);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (i + u * nt < we * RPW * BNW) gy[i + u * nt] = a[u];
    }
    __syncthreads();
    const int at = min(g, RPW - 1);  // lanes past the last chain repeat one; they store nothing
    for (; q < per; q += nw) {
        const int row = (at * per + q) * BNL + r;
        T t = row < nrows ? ysh[row] : T(0);
        while (k1 > 0) {
            const int m = min(k1, B);
            T cur[B][BNW];
#pragma unroll
            for (int u = 0; u < B; u++)
#pragma unroll
                for (int l = 0; l < BNW; l++) cur[u][l] = v[u][l];
            const T *gk = gy + ((s0 + k1 - B) * RPW + at) * BNW;  // used from the first slot in use on
            const int next = k1 + B;
            if (k1 < width) load(s0, next);
            sub_slots<BNW, B>(t, cur, gk, RPW * BNW, m);
            k1 = k1 < width ? next : 0;
        }
        if (g < RPW && row < nrows) ysh[row] = t;
        if (q + nw < per) {
            for (int k = q; k < q + nw; k++) s0 += wd[k];
            width = wd[q + nw];
            k1 = width > 0 ? (width - 1) % B + 1 : 0;
            if (k1 > 0) load(s0, k1);
        }
    }
    __syncthreads();
    if (w == 0) {
        const int base = at * BNL;
        for (int st = 0; st < per; st++) {
            const int qq = UPPER ? per - 1 - st : st;
            int i0 = 0;
            for (int k = 0; k < qq; k++) i0 += wd[per + k];
            const int row = (at * per + qq) * BNL + r;
            const bool live = g < RPW && row < nrows;
            T t = live ? ysh[row] : T(0);
            const int m = wd[per + qq];
#pragma unroll 1
            for (int k = 0; k < m; k++) {
                const int c = lc[(i0 + k) * RPW + at], rel0 = c - qq * BNL;
                const bool inside = !UPPER && c >= 0 && rel0 >= 0 && rel0 < BNL;
                const bool any = !UPPER && __any_sync(0xffffffffu, inside);
#pragma unroll
                for (int l = 0; l < BNW; l++) {
                    const T vv = val[((size_t)(i0 + k) * BNW + l) * 32 + lane];
                    const T yy = c >= 0 ? ysh[at * per * BNL + c + l] : T(0);
                    T tout = t;
                    if (!any || __any_sync(0xffffffffu, !inside && c >= 0)) tout = t - vv * yy;
                    if (any) {
                        const int rel = inside ? rel0 + l : 0;
                        const T a0 = __shfl_sync(0xffffffffu, t, base + rel);
                        const T t0 = t - vv * a0;
                        const T a1 = __shfl_sync(0xffffffffu, t0, base + rel);  // y[col] after its own pair
                        const T t1 = (r >> 1) > (rel >> 1) ? t - vv * a1 : t0;
                        if (inside) tout = t1;
                    }
                    t = tout;
                }
            }
            if (UPPER) {
#pragma unroll
                for (int c = BNL - 1; c >= 0; c--) {
                    const T dc = diag[((size_t)qq * BNL + c) * 32 + lane];
                    if (r == c) t *= dc;
                    const T a = __shfl_sync(0xffffffffu, t, base + c);
                    if (r < c) t -= dc * a;
                }
            }
            if (live) ysh[row] = t;
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = tid; i < nrows; i += nt) y[r0 + i] = ysh[i];
}

#define SENK_ILUB_SHAPES(X) X(1, 1) X(2, 1) X(2, 2) X(3, 3) X(4, 1) X(4, 2) X(4, 4) X(8, 1) X(8, 2)

bool shape_supported(int bnl, int bnw)
{
#define X(R, C) if (bnl == R && bnw == C) return true;
    SENK_ILUB_SHAPES(X)
#undef X
    return false;
}

int lanes_of(int bnl) { return bnl <= 1 ? 1 : bnl <= 2 ? 2 : bnl <= 4 ? 4 : bnl <= 8 ? 8 : bnl <= 16 ? 16 : 32; }

// Checks one factor against the schedule: every column a block row reads from
// outside itself must be final when the block row runs (an earlier phase, or
// an earlier block row of its own chain). The reference would race otherwise.
void check_factor(bool upper, int nbr, int bnl, int bnw, const int *bcind, const int *brptr,
                  const std::vector<int2> &chains, const std::vector<int> &phase_chains, const char *name)
{
    const int nbc = nbr * bnl / bnw, brem = bnl / bnw;
    SENK_REQUIRE(brptr[0] == 0, std::string(name) + ": brptr[0] must be 0");
    for (int br = 0; br < nbr; br++) {
        SENK_REQUIRE(brptr[br + 1] >= brptr[br], std::string(name) + ": brptr not monotonic");
        for (int j = brptr[br]; j < brptr[br + 1]; j++)
            SENK_REQUIRE(bcind[j] >= 0 && bcind[j] < nbc, std::string(name) + ": block column out of range");
        if (upper) {
            SENK_REQUIRE(brptr[br + 1] - brptr[br] >= brem,
                         std::string(name) + ": block row without its diagonal square");
            for (int m = 0; m < brem; m++)
                SENK_REQUIRE(bcind[brptr[br] + m] == br * brem + m,
                             std::string(name) + ": the leading blocks of a row must be its diagonal square");
        }
    }
    // done[br]: 2 = finished in an earlier phase; 1 = finished earlier in the
    // chain being checked
    std::vector<unsigned char> done(nbr, 0);
    const int P = (int)phase_chains.size() - 1;
    for (int pi = 0; pi < P; pi++) {
        const int p = upper ? P - 1 - pi : pi;
        for (int c = phase_chains[p]; c < phase_chains[p + 1]; c++) {
            const int2 ch = chains[c];
            for (int q = 0; q < ch.y; q++) {
                const int br = upper ? ch.x + ch.y - 1 - q : ch.x + q;
                const int j0 = brptr[br] + (upper ? brem : 0);
                for (int j = j0; j < brptr[br + 1]; j++) {
                    for (int l = 0; l < bnw; l++) {
                        const int col = bcind[j] * bnw + l, cbr = col / bnl;
                        if (cbr == br) {
                            SENK_REQUIRE(!upper, std::string(name) + ": U block right of the diagonal square "
                                                                     "reaches into its own block row");
                            continue;
                        }
                        SENK_REQUIRE(done[cbr] != 0, std::string(name) + ": block row " + std::to_string(br) +
                                                         " reads row " + std::to_string(col) +
                                                         " before the schedule has finished it");
                    }
                }
                done[br] = 1;
            }
            // rows of this chain may not be read by the other chains of the phase
            for (int q = 0; q < ch.y; q++) done[ch.x + q] = 0;
        }
        for (int c = phase_chains[p]; c < phase_chains[p + 1]; c++)
            for (int q = 0; q < chains[c].y; q++) done[chains[c].x + q] = 2;
    }
    for (int br = 0; br < nbr; br++) SENK_REQUIRE(done[br] == 2, std::string(name) + ": block row not scheduled");
}

}  // namespace

template <typename T>
void IlubPlan<T>::build(int N, int bnl_, int bnw_, const T *blval, const int *blcind, const int *blrptr,
                        const T *buval, const int *bucind, const int *burptr, const int *cptr, int cnum, int bsize,
                        cudaStream_t s)
{
    SENK_REQUIRE(shape_supported(bnl_, bnw_), "ILUB block shape " + std::to_string(bnl_) + "x" +
                                                  std::to_string(bnw_) +
                                                  " is not built (1x1 2x1 2x2 3x3 4x1 4x2 4x4 8x1 8x2)");
    SENK_REQUIRE(N > 0 && N % bnl_ == 0, "N must be a multiple of bnl");
    SENK_REQUIRE(blval && blcind && blrptr && buval && bucind && burptr, "null BCSR factor array");
    n = N;
    bnl = bnl_;
    bnw = bnw_;
    nbr = N / bnl;
    std::vector<int2> ch;
    phase_chains.assign(1, 0);
    if (cptr) {
        SENK_REQUIRE(cnum > 0 && bsize > 0 && bsize % bnl == 0, "ABMC bsize must be a positive multiple of bnl");
        SENK_REQUIRE(cptr[0] == 0, "cptr[0] must be 0");
        const int per = bsize / bnl;
        for (int c = 0; c < cnum; c++) {
            SENK_REQUIRE(cptr[c + 1] >= cptr[c], "cptr not monotonic");
            for (int blk = cptr[c]; blk < cptr[c + 1]; blk++) {
                const long long first = (long long)blk * per;
                SENK_REQUIRE(first < nbr, "colour block beyond N");
                ch.push_back(make_int2((int)first, (int)std::min<long long>(per, nbr - first)));
            }
            phase_chains.push_back((int)ch.size());
        }
    } else {
        ch.push_back(make_int2(0, nbr));
        phase_chains.push_back(1);
    }
    check_factor(false, nbr, bnl, bnw, blcind, blrptr, ch, phase_chains, "ILUB L factor");
    check_factor(true, nbr, bnl, bnw, bucind, burptr, ch, phase_chains, "ILUB U factor");
    lblocks = blrptr[nbr];
    ublocks = burptr[nbr];
    const size_t bs = (size_t)bnl * bnw;
    status.alloc(1);
    SENK_CUDA(cudaMemsetAsync(status.p, 0, sizeof(int), s));
    auto put = [s](auto &buf, const auto *h, size_t count) {
        buf.alloc(count);
        buf.upload(h, count, s);
    };
    put(lval, blval, (size_t)lblocks * bs);
    put(lcind, blcind, (size_t)lblocks);
    put(lrptr, blrptr, (size_t)nbr + 1);
    put(uval, buval, (size_t)ublocks * bs);
    put(ucind, bucind, (size_t)ublocks);
    put(urptr, burptr, (size_t)nbr + 1);
    per = cptr ? bsize / bnl : 0;
    sliced = cptr && per <= kBlMaxSteps && build_slices(false, blcind, blrptr, ch, s) &&
             build_slices(true, bucind, burptr, ch, s);
    if (!sliced) {
        ls = Slices();
        us = Slices();
    }
    if (sliced) {  // the slices hold everything the sweeps read
        SENK_CUDA(cudaStreamSynchronize(s));
        for (auto *v : {&lval, &uval}) v->release();
        for (auto *v : {&lcind, &lrptr, &ucind, &urptr}) v->release();
    } else {
        put(chains, ch.data(), ch.size());
    }
    SENK_CUDA(cudaStreamSynchronize(s));  // the host vectors go out of scope
}

// Groups, widths and the slice layout of one factor (k_ilub_slices), filled on
// the device from the BCSR arrays uploaded before. False when a group does not
// fit the shared memory or a block row's blocks outside its chain do not come
// first.
template <typename T>
bool IlubPlan<T>::build_slices(bool upper, const int *bcind, const int *brptr, const std::vector<int2> &ch,
                               cudaStream_t s)
{
    const int rpw = 32 / bnl, brem = bnl / bnw;
    const int P = (int)phase_chains.size() - 1;
    Slices &F = upper ? us : ls;
    std::vector<BlGroup> gd;
    F.launches.clear();
    for (int pi = 0; pi < P; pi++) {  // colours in processing order
        const int p = upper ? P - 1 - pi : pi;
        const int before = (int)gd.size();
        for (int c = phase_chains[p]; c < phase_chains[p + 1]; c += rpw)
            gd.push_back({ch[c].x, std::min(rpw, phase_chains[p + 1] - c), 0, 0});
        if ((int)gd.size() > before) F.launches.push_back({before, (int)gd.size(), 0});
    }
    const int ng = (int)gd.size();
    // at any width: 3x3 blocks, 10.5 to 28.9 groups to an SM and colour (80^3 to 112^3
    // nodes), one FP64 application and 20 GCR iterations against k_ilub_sweep's:
    // 0.43 : 0.62 ms and 17.3 : 20.5 at 10.5, 0.57 : 0.73 and 22.6 : 25.5 at 14, 0.72 :
    // 0.75 and 28.7 : 28.6 at 18.2, 0.77 : 1.07 and 31.4 : 37.0 at 20.6, 1.03 : 1.45 and
    // 42.9 : 51.2 at 28.9
    std::vector<uint16_t> widths((size_t)ng * 2 * per, 0);
    bool fits = true;
#pragma omp parallel for schedule(static) reduction(&& : fits)
    for (int g = 0; g < ng; g++)
        for (int c = 0; c < gd[g].nch; c++)
            for (int q = 0; q < per; q++) {
                const int br = gd[g].row0 + c * per + q, first = (gd[g].row0 + c * per) * bnl;
                if (br >= nbr) continue;
                int we = 0, wi = 0;
                const int a = brptr[br] + (upper ? brem : 0), e = brptr[br + 1];
                for (int i = a; i < e; i++) {  // in the sweep's order
                    const int col = bcind[upper ? e - 1 - (i - a) : i] * bnw;
                    if (col >= first && col < first + per * bnl) {
                        wi++;
                    } else {
                        we++;
                        fits = fits && wi == 0;  // external blocks come first
                    }
                }
                uint16_t *w = &widths[(size_t)g * 2 * per];
                fits = fits && we < 65536 && wi < 65536;
                w[q] = (uint16_t)std::max<int>(w[q], we);
                w[per + q] = (uint16_t)std::max<int>(w[per + q], wi);
            }
    if (!fits) return false;
    long long ext = 0, blob = 0;
    std::vector<size_t> smem(ng);
    for (int g = 0; g < ng; g++) {
        const uint16_t *w = &widths[(size_t)g * 2 * per];
        int we = 0, wi = 0;
        for (int q = 0; q < per; q++) {
            we += w[q];
            wi += w[per + q];
        }
        const BlParts parts = bl_parts(per, we, wi, rpw, bnl, bnw, upper, sizeof(T));
        gd[g].ext = (int)ext;
        gd[g].blob = (int)blob;
        ext += we;
        blob += parts.end / 16;
        smem[g] = parts.end + ((size_t)rpw * kBlMaxSteps * bnl + (size_t)we * rpw * bnw) * sizeof(T);
        if (smem[g] > kBlMaxSmem || ext >= (1 << 30) || blob >= (1 << 30)) return false;
    }
    gd.push_back({0, 0, (int)ext, (int)blob});
    for (size_t k = 0; k < F.launches.size(); k++) {
        auto &L = F.launches[k];
        L.order = (int)std::min<size_t>(k, 2);
        for (int g = L.g0; g < L.g1; g++) L.smem = std::max(L.smem, smem[g]);
    }
    F.groups.alloc(gd.size());
    F.groups.upload((const int4 *)gd.data(), gd.size(), s);
    F.ext.alloc(std::max<size_t>((size_t)ext * bnw * 32, 1));
    F.blob.alloc(std::max<size_t>((size_t)blob * 16, 16));
    DevBuf<uint16_t> dw(widths.size());
    dw.upload(widths.data(), widths.size(), s);
    const BlGroup *dg = (const BlGroup *)F.groups.p;
#define X(R, C)                                                                                                  \
    if (bnl == R && bnw == C) {                                                                                  \
        if (upper) {                                                                                             \
            k_ilub_fill<T, R, C, true><<<ng, 32 * per, 0, s>>>(dg, dw.p, per, nbr, uval.p, ucind.p, urptr.p, F.ext.p, \
                                                               F.blob.p);                                        \
            SENK_CUDA(cudaFuncSetAttribute(k_ilub_slices<T, R, C, true>,                                         \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlMaxSmem));       \
        } else {                                                                                                 \
            k_ilub_fill<T, R, C, false><<<ng, 32 * per, 0, s>>>(dg, dw.p, per, nbr, lval.p, lcind.p, lrptr.p,    \
                                                                F.ext.p, F.blob.p);                              \
            SENK_CUDA(cudaFuncSetAttribute(k_ilub_slices<T, R, C, false>,                                        \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlMaxSmem));       \
        }                                                                                                        \
    } else
    SENK_ILUB_SHAPES(X)
#undef X
    throw ArgError("unsupported ILUB block shape");
    SENK_LAUNCH_CHECK();
    SENK_CUDA(cudaStreamSynchronize(s));  // the widths go out of scope
    return true;
}

template <typename T>
void IlubPlan<T>::sweep(bool upper, const T *x, T *y, cudaStream_t s, const int *gate) const
{
    if (sliced) {
        const Slices &F = upper ? us : ls;
        for (const auto &L : F.launches) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(L.g1 - L.g0);
            cfg.blockDim = dim3(32 * std::min(per, 8));
            cfg.dynamicSmemBytes = L.smem;
            cfg.stream = s;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
#define X(R, C)                                                                                                \
    if (bnl == R && bnw == C)                                                                                  \
        SENK_CUDA(cudaLaunchKernelEx(&cfg, upper ? k_ilub_slices<T, R, C, true> : k_ilub_slices<T, R, C, false>, \
                                     (const BlGroup *)F.groups.p, L.g0, per, n, (const T *)F.ext.p,             \
                                     (const uint4 *)F.blob.p, x, y, gate, status.p, L.order));                  \
    else
            SENK_ILUB_SHAPES(X)
#undef X
            throw ArgError("unsupported ILUB block shape");
        }
        SENK_LAUNCH_CHECK();
        return;
    }
    const int P = (int)phase_chains.size() - 1;
    const int G = lanes_of(bnl);
    for (int pi = 0; pi < P; pi++) {
        const int p = upper ? P - 1 - pi : pi;
        const int c0 = phase_chains[p], nch = phase_chains[p + 1] - c0;
        if (nch == 0) continue;
        const long long lanes = (long long)nch * G;
        const int threads = (int)std::min<long long>(kThreads, (lanes + 31) / 32 * 32);
        const int grid = ceil_div(lanes, threads);
#define X(R, C)                                                                                               \
    if (bnl == R && bnw == C) {                                                                               \
        if (upper)                                                                                            \
            k_ilub_sweep<T, R, C, true><<<grid, threads, 0, s>>>(uval.p, ucind.p, urptr.p, chains.p + c0, nch, x, \
                                                                 y, gate);                                    \
        else                                                                                                  \
            k_ilub_sweep<T, R, C, false><<<grid, threads, 0, s>>>(lval.p, lcind.p, lrptr.p, chains.p + c0, nch, \
                                                                  x, y, gate);                                \
    } else
        SENK_ILUB_SHAPES(X)
#undef X
        throw ArgError("unsupported ILUB block shape");
        SENK_LAUNCH_CHECK();
    }
}

template <typename T>
void IlubPlan<T>::check_status(cudaStream_t s) const
{
    int h = 0;
    SENK_CUDA(cudaMemcpyAsync(&h, status.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    SENK_CUDA(cudaStreamSynchronize(s));
    if (!h) return;
    // reported once: the next sweep starts clean
    SENK_CUDA(cudaMemsetAsync(status.p, 0, sizeof(int), s));
    SENK_CUDA(cudaStreamSynchronize(s));
    throw CudaError{cudaErrorLaunchTimeout, "ILUB sweep: a TMA copy of a group's factor block did not complete", __FILE__,
                    __LINE__};
}

template <typename T>
long long IlubPlan<T>::apply_bytes() const
{
    const long long vb = sizeof(T), bs = (long long)bnl * bnw;
    // blocks (values + block column) and block row pointers of both factors;
    // x read, y written by L, read and written by U
    return (lblocks + ublocks) * (bs * vb + 4) + 2LL * (nbr + 1) * 4 + 4LL * n * vb;
}

template struct IlubPlan<double>;
template struct IlubPlan<float>;

void learned_apply(void *net, const void *sys, const double *v, double *out, cudaStream_t s);

template <typename T>
void System<T>::precondition(const T *v, T *out, const int *gate)
{
    precondition_base(v, out, gate);
    if constexpr (std::is_same<T, double>::value) {
        if (learned) learned_apply(learned, this, v, out, stream);
    }
}

template <typename T>
void System<T>::precondition_base(const T *v, T *out, const int *gate)
{
    if (pcb) pcb->apply(v, out, stream, gate);
    else if (pc) pc->apply(v, out, stream, gate);
    else
        k_elementwise<T, 4><<<stream_grid(n, kThreads, 8), kThreads, 0, stream>>>(T(0), nullptr, 1.0, T(0), v, out,
                                                                                  nullptr, n, gate);
    SENK_LAUNCH_CHECK();
}

template <typename T>
void System<T>::check_pc() const
{
    if (pc) pc->check_status(stream);
    if (pcb) pcb->check_status(stream);
}

template void System<double>::precondition(const double *, double *, const int *);
template void System<float>::precondition(const float *, float *, const int *);
template void System<double>::precondition_base(const double *, double *, const int *);
template void System<float>::precondition_base(const float *, float *, const int *);
template void System<double>::check_pc() const;
template void System<float>::check_pc() const;

}  // namespace senkgpu
