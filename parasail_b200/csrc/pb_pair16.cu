/*
 * pb_pair16.cu -- global (NW), semi-global (SG) and local (SW) alignment of
 * batches of independent pairs in packed int16x2 lanes, with statistics
 * (matches, similar, length) and paths from a traceback over checkpoints.
 *
 * Inter-task schedule: one thread aligns one pair; a warp takes a task of
 * 32 pairs of like size (items sorted by passes and columns); a persistent
 * grid pulls tasks in order of cost. The query is processed in passes of
 * 2 x 16 rows lag-packed in int16x2 words, as in the Smith-Waterman
 * database kernel (pb_sw16.cu): the low half of every register holds strip
 * A (rows r0..r0+15) at column j, the high half strip B (rows r0+16..r0+31)
 * at column j-1, so strip B reads strip A's bottom row from the previous
 * iteration. A pass hands its bottom row (H and F) to the next pass through
 * the warp's buffer laid out [column][lane] (one 128-byte transaction per
 * warp access). Each lane (pairs mode) or each warp (all 32 pairs of the
 * task share a query) stages the scores of the pass's 32 rows against every
 * alphabet letter in shared memory as int8 (a column's 16 + 16 scores are
 * two 16-byte loads expanded by sign-extending byte permutes).
 *
 * Semantics are the reference's serial dynamic programs (src/sw.c:102-158,
 * src/nw.c:102-156, src/sg.c:117-242 and the _stats twins), which its
 * striped and scan kernels reproduce for every non-saturated result:
 *   F(i,j) = max(H(i-1,j) - open, F(i-1,j) - gap)    vertical gap
 *   E(i,j) = max(H(i,j-1) - open, E(i,j-1) - gap)    horizontal gap
 *   H(i,j) = max(H(i-1,j-1) + s(i,j), E(i,j), F(i,j)) (SW: and 0)
 * with the boundaries of src/nw.c:102-120 and src/sg.c:117-143, and the end
 * rules of src/sw.c:150-158 (first maximum in column-major order) and
 * src/sg.c:160-242.
 *
 * Exactness in 16 bits. An item runs here only when sound bounds keep
 * every value it computes, padded rows included, inside int16 with the
 * differences below as well: every H is at most max(matrix) x (min(rows,
 * cols) + 1), and at least -(3 open + (rows32 + cols + 2) gap) + min(matrix)
 * (a path of two gaps reaches any cell); E and F are at least H - open.
 * "-inf" is a per-lane value NEG = LB - open - 1, which no gap opened from
 * a real cell can tie. Items outside the bounds run on the exact 32-bit
 * kernel instead.
 *
 * Statistics. The reference's statistics recurrence (src/sw_stats.c:
 * 204-264, src/nw_stats.c:190-218, src/sg_stats.c:227-265) carries, with
 * every H, E and F, the counts of the one path its tie rules select: the
 * gap source by strict > (open only when H - open > E - gap), the cell
 * source diagonal, then F, then E; SW restarts at H <= 0 and the boundary
 * cells carry 0. Those counts are the counts along that path, which four
 * decisions per cell define: not-diagonal (H > H_diag + s), not-F (H > F), E
 * opened and F opened. The forward kernel leaves checkpoints instead of the
 * decisions -- every pass's bottom row, and its column state every p16_ck
 * columns -- and the traceback (k_p16_trace) recomputes only the blocks that
 * the path from the end cell crosses, adding 1 to length per step and, on
 * diagonal steps, the match and positive-score indicators; in SW it stops
 * where the running H value (the end score minus the steps walked) reaches
 * 0, in NW/SG at the boundary.
 */
#include <cstdio>
#include <cstdint>
#include <climits>
#include <cstring>
#include <algorithm>
#include <vector>

#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <cuda/std/functional>
#include <dlfcn.h>
#include <mutex>
#include <string>

#include "pb_cuda.h"
#include "pb_kernels.cuh"
#include "pb_resolve.h"
#include "pb_slices.h"

namespace pb {

static constexpr int P16_R = 16;              /* rows per strip; two strips per pass */
static constexpr int P16_PASS = 2 * P16_R;
static constexpr int P16_ROW = 48;            /* bytes between two letters' scores in a shared slice */

static constexpr int P16_TR_WARPS = 2;        /* warps per block of the traceback */
/* Checkpoints of a task (one lane's words 32 apart): per pass its bottom row,
 * p16_cols words (entry c + 1: H low and F high at column c), and per pass
 * and block of p16_ck columns after the first the state before the block's
 * first iteration: H and E of the 16 register rows, F of the last one, and
 * the next diagonal. */
static constexpr int P16_CK_U4 = P16_R / 2 + 1;
/* Columns per block. A path that crosses every pass recomputes blocks in step
 * with the 31 others of its warp, a whole block each time: 16 (1 M reads, NW:
 * traceback 8.7 -> 7.0 ms, forward pass 10.3 -> 10.4). Short local paths
 * cross few blocks, and the column states' traffic counts: 32 (all against
 * all: forward pass 72.7 ms, 78.2 with 16). */
__host__ __device__ constexpr int p16_ck(int alg) { return alg == PB_SW ? 32 : 16; }
__host__ __device__ __forceinline__ int p16_ck_blocks(int alg, int wmax) { return (p16_cols(wmax) - 1) / p16_ck(alg); }
/* in words */
__device__ __forceinline__ size_t p16_ck_row(int wmax, int pass, int entry)
{
    return ((size_t)pass * p16_cols(wmax) + entry) * 32;
}
/* in uint4 from the task's first */
__host__ __device__ __forceinline__ size_t p16_ck_col(int alg, int npass, int wmax, int pass, int block)
{
    return (size_t)npass * p16_cols(wmax) * 8 + ((size_t)pass * p16_ck_blocks(alg, wmax) + block) * P16_CK_U4 * 32;
}

/* the bit of query row i of a block's direction bits (row i of its pass): the
 * byte by the row's parity and strip, the bit by its pair of rows */
__device__ __forceinline__ int p16_bit(int i) { return ((i & 1) * 2 + ((i >> 4) & 1)) * 8 + ((i & 15) >> 1); }

__device__ __forceinline__ uint32_t p16_prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

/* byte K of a (low half) and of b (high half), sign-extended to int16x2 */
template <int K>
__device__ __forceinline__ uint32_t p16_pair(uint32_t a, uint32_t b)
{
    constexpr uint32_t sel = (K) | ((K | 8) << 4) | ((4 + K) << 8) | (((4 + K) | 8) << 12);
    return p16_prmt(a, b, sel);
}

__device__ __forceinline__ uint32_t p16_splat(int v) { return ((uint32_t)(uint16_t)v) | ((uint32_t)(uint16_t)v << 16); }
__device__ __forceinline__ int p16_lo(uint32_t x) { return (int)(int16_t)(x & 0xffffu); }
__device__ __forceinline__ int p16_hi(uint32_t x) { return (int)(int16_t)(x >> 16); }

/* The bounds of one item (see the file comment). */
struct P16Bounds {
    int lb, ub;
};

__host__ __device__ __forceinline__ P16Bounds p16_bounds(int alg, int rows, int cols, int open, int gap,
                                                         int mmax, int mmin)
{
    P16Bounds b;
    const long long r32 = ((long long)rows + 31) / 32 * 32;
    const long long mn = mmin < 0 ? mmin : 0, mx = mmax > 0 ? mmax : 0;
    const long long ub = mx * ((rows < cols ? rows : cols) + 1);
    long long lb = alg == PB_SW ? mn : -(3LL * open + (r32 + cols + 2) * (long long)gap) + mn;
    b.lb = lb < INT_MIN / 2 ? INT_MIN / 2 : (int)lb;
    b.ub = ub > INT_MAX / 2 ? INT_MAX / 2 : (int)ub;
    return b;
}

__host__ __device__ __forceinline__ bool p16_fits(const P16Bounds &b, int open, int gap)
{
    return (long long)b.ub - b.lb + open + gap + 1 <= 32000;
}

/* boundary H of row -1 (column j) and column -1 (row i); H(-1,-1) = 0 */
__device__ __forceinline__ int p16_top(int alg, int sgf, int j, int open, int gap)
{
    if (alg == PB_SW || (alg == PB_SG && (sgf & PB_S2_BEG))) return 0;
    return -open - j * gap;
}

__device__ __forceinline__ int p16_left(int alg, int sgf, int i, int open, int gap)
{
    if (i < 0) return 0;
    if (alg == PB_SW || (alg == PB_SG && (sgf & PB_S1_BEG))) return 0;
    return -open - i * gap;
}

struct P16Best {
    int score, i, j;
};

/*
 * One task (32 items) per warp at a time. SHARED: every lane of a task has
 * the same query (its scores are staged once per warp); else every lane
 * stages its own. CKPT: leave the checkpoints that the traceback restarts
 * from (p16_ck_row, p16_ck_col). ENDS: compute score and ends (off for the
 * FASTSTATS prefix pass, whose ends are known). BIAS (open >= gap, every
 * score + open inside int8): H registers and boundaries hold H - open, staged
 * scores s + open, so the gap sources need no add, and F of the next row is
 * max(F - gap, max(H_diag + s, E) - open).
 *
 * What bounds it: the ALU pipe at half rate (maxima, three-operand DPX, byte
 * permutes), with the packed adds on the FMA pipe beside it: 5 ALU and 1 FMA
 * operations per row of two cells. As in k_sw16, four columns run without a
 * branch each, targets are read by words (the code check of a byte load
 * waited for the load in every column), and the staged scores are laid out
 * so that 16-byte loads fall on all bank groups: [letter][48 bytes] per
 * warp, or [letter][strip][lane] x 16 bytes. The checkpoints add 8.5 bytes
 * per column and lane (0.27 per cell), where the direction bits of every
 * cell took 0.5 bytes and twice the operations.
 * 1 M DNA reads, NW: 29.3 ms with direction bits, now 10.3 ms with
 * checkpoints; 524 k protein pairs all against all: score pass 93.5 -> 72.7
 * ms with checkpoints (65.7 without).
 */
template <int ALG, bool CKPT, bool ENDS, bool SHARED, int WARPS, bool BIAS>
__global__ void __launch_bounds__(WARPS * 32, (WARPS == 8 ? 2 : 3))
k_p16(P16Params p, const int *__restrict__ tlist, int ntl, int *counter)
{
    extern __shared__ __align__(16) int8_t s_mem[];
    constexpr int LETTER = SHARED ? P16_ROW : 1024, STRIP = SHARED ? 16 : 512;
    const int L = p.nletters;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int open = p.open, gap = p.gap, sgf = p.sgflags;
    const int bias = BIAS ? open : 0;
    /* shared memory: [matrix L x L int8, padded to 16] [per-warp score slices] */
    const int mat_bytes = p.mat8 ? ((L * L + 15) & ~15) : 0;
    int8_t *s_mat = s_mem;
    int8_t *wslice = s_mem + mat_bytes + wid * L * LETTER;
    int8_t *sl = wslice + (SHARED ? 0 : lane * 16);
    if (p.mat8)
        for (int k = threadIdx.x; k < L * L; k += blockDim.x) s_mat[k] = (int8_t)(p.mat8[k] + bias);
    __syncthreads();

    /* pass boundary: entry c + 1 is strip B's bottom row at column c, H low
     * and F high */
    uint32_t *buf = p.scratch + (size_t)(blockIdx.x * WARPS + wid) * (size_t)(p.maxlen + 8) * 32 + lane;
    /* SW ends: this thread's copies of its strips' best columns */
    uint4 *save = ENDS && ALG == PB_SW ? p.colsave + ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * (P16_R / 2)
                                       : nullptr;
    const uint32_t gO = p16_splat(-open), gE = p16_splat(-gap);
    const uint32_t b4 = 0x01010101u * (uint32_t)(uint8_t)bias;
    const uint32_t big4 = 0x01010101u * (uint32_t)(0x80 - L);
    const int nwarps_total = gridDim.x * WARPS;
    bool first = true;
    for (;;) {
        int k;
        if (first) {
            k = blockIdx.x + gridDim.x * wid;
            first = false;
        } else {
            if (lane == 0) k = nwarps_total + atomicAdd(counter, 1);
            k = __shfl_sync(0xffffffffu, k, 0);
        }
        if (k >= ntl) break;
        const int task = tlist[k];
        const int s = task * 32 + lane;
        const bool valid = s < p.nitems && p.order[s] >= 0;
        const int item = valid ? p.order[s] : 0;
        const int rows = valid ? p.rows[item] : 0;
        const int cols = valid ? p.cols[item] : 0;
        const int wmax = p.task_wmax[task];
        const int npass = p.task_npass[task];
        const int ti = p.nt ? item % p.nt : item;
        const uint8_t *tseq = p.targets + (valid ? p.toff[ti] : 0);
        /* query source */
        const uint8_t *qseq = nullptr;
        const int8_t *prof8 = nullptr;
        int lp = 0;
        if (p.mat8) {
            qseq = p.qall + (valid ? p.qoff[item] : 0);
        } else {
            /* an invalid lane (a task's padding) takes the task's query:
             * in the shared variant every lane writes part of the slice
             * from its own profile pointer */
            const int qitem = valid ? item : p.order[task * 32];
            const ProfDesc pd = p.profs[p.nt ? qitem / p.nt : 0];
            prof8 = pd.prof8;
            lp = pd.lp;
        }
        int rmax = rows;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
        const uint8_t *qseq0 = SHARED && p.mat8 ? p.qall + p.qoff[p.order[task * 32]] : nullptr;
        const P16Bounds bd = p16_bounds(ALG, rows, cols, open, gap, p.mmax, p.mmin);
        const int negv = bd.lb - open - 1;
        const uint32_t NEG = p16_splat(negv);
        /* the task's checkpoints: rows (entry c + 1 of a pass: its bottom row at
         * column c), then columns */
        uint32_t *ckr = CKPT ? reinterpret_cast<uint32_t *>(p.ckpt + p.task_ckpt[task]) + lane : nullptr;
        uint4 *ckc = CKPT ? p.ckpt + p.task_ckpt[task] + p16_ck_col(ALG, npass, wmax, 0, 0) + lane : nullptr;
        int status = 0;

        /* end tracking */
        P16Best best = {0, 0, 0};
        int lc_h = INT_MIN, lc_i = -1;       /* SG: last column over rows < rows - 1 */
        int lr_h = INT_MIN, lr_j = -1;       /* SG: last row */
        int corner = 0;
        const int ilast = rows - 1;
        const int p_last = ilast >> 5, half_last = (ilast >> 4) & 1, r_last = ilast & 15;

        for (int pass = 0; pass < npass; ++pass) {
            const int r0 = pass * P16_PASS;
            /* scores (BIAS: + open) of this pass's 32 rows against every
             * letter: once per warp (shared query) or once per lane; rows past
             * the query (past the task's longest in shared pairs mode) score 0 */
            if (SHARED) {
                __syncwarp();
                if (p.mat8) {
                    const int i = r0 + lane;
                    uint32_t c = 255u;               /* past the query */
                    if (i < rmax) {
                        c = qseq0[i];
                        if (c >= (uint32_t)L) { c = 0; status |= PB_ST_BADCODE; }
                    }
                    for (int a = 0; a < L; ++a)
                        wslice[a * LETTER + lane] = c == 255u ? (int8_t)bias : s_mat[a * L + c];
                } else {
                    for (int x = lane; x < 2 * L; x += 32) {
                        const int a = x >> 1, h = x & 1;
                        int4 v = *reinterpret_cast<const int4 *>(prof8 + (size_t)a * lp + r0 + 16 * h);
                        if (BIAS) {
                            v.x = (int)__vadd4((uint32_t)v.x, b4); v.y = (int)__vadd4((uint32_t)v.y, b4);
                            v.z = (int)__vadd4((uint32_t)v.z, b4); v.w = (int)__vadd4((uint32_t)v.w, b4);
                        }
                        *reinterpret_cast<int4 *>(wslice + a * LETTER + 16 * h) = v;
                    }
                }
            } else {
                /* (pairs mode: a task of the database mode shares its query) */
                uint32_t qc[8];
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    uint32_t word = 0;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const int i = r0 + 4 * w + b;
                        uint32_t c = 255u;           /* past the query */
                        if (i < rows) {
                            c = qseq[i];
                            if (c >= (uint32_t)L) { c = 0; status |= PB_ST_BADCODE; }
                        }
                        word |= c << (8 * b);
                    }
                    qc[w] = word;
                }
                for (int a = 0; a < L; ++a) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t word[4];
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            word[w] = 0;
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                const uint32_t c = (qc[4 * h + w] >> (8 * b)) & 0xffu;
                                const uint32_t v = c == 255u ? (uint32_t)(uint8_t)bias
                                                             : (uint32_t)(uint8_t)s_mat[a * L + c];
                                word[w] |= v << (8 * b);
                            }
                        }
                        *reinterpret_cast<uint4 *>(sl + a * LETTER + h * STRIP) =
                            make_uint4(word[0], word[1], word[2], word[3]);
                    }
                }
            }
            __syncwarp();

            /* initial state: column -1 */
            uint32_t H[P16_R], E[P16_R];
#pragma unroll
            for (int r = 0; r < P16_R; ++r) {
                const int la = p16_left(ALG, sgf, r0 + r, open, gap) - bias;
                const int lb2 = p16_left(ALG, sgf, r0 + P16_R + r, open, gap) - bias;
                H[r] = (uint32_t)(uint16_t)la | ((uint32_t)(uint16_t)lb2 << 16);
                E[r] = NEG;
            }
            uint32_t dg = (uint32_t)(uint16_t)(p16_left(ALG, sgf, r0 - 1, open, gap) - bias);
            uint32_t prev_h = (uint32_t)(uint16_t)(p16_left(ALG, sgf, r0 + P16_R - 1, open, gap) - bias);
            uint32_t prev_f = NEG & 0xffffu;
            /* the row above: row -1 (H by the boundary, F = -inf) in the first
             * pass, else the previous pass's bottom row, loaded four columns
             * ahead (this pass overwrites entry j at column j) */
            const bool top = pass == 0;
            uint32_t vtop = p16_prmt((uint32_t)(uint16_t)(p16_top(ALG, sgf, 0, open, gap) - bias), NEG, 0x5410u);
            const uint32_t top_step = (ALG == PB_SW || (ALG == PB_SG && (sgf & PB_S2_BEG))) ? 0u
                                                                                           : (uint32_t)(uint16_t)(-gap);
            const uint32_t vnone = p16_prmt(0u, NEG, 0x5410u);
            const int rd = top ? 0 : wmax;
            const uint32_t *in_row = CKPT ? ckr + (top ? 0 : p16_ck_row(wmax, pass - 1, 0)) : buf;
            uint32_t v_n[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) v_n[x] = x < rd ? __ldcg(in_row + (x + 1) * 32) : vnone;
            const uint32_t *in_at = in_row + 5 * 32;
            uint32_t *out_at = CKPT ? ckr + p16_ck_row(wmax, pass, 0) : buf;
            P16Best sa = {0, -1, -1}, sb = {0, -1, -1};
            /* SW: what a column maximum has to pass, as in k_sw16 */
            uint32_t sbest = p16_splat(max(best.score - 1, 0) - bias);
            const bool more = pass + 1 < npass;
            const bool lastpass = ENDS && ALG != PB_SW && pass == p_last;
            const int8_t *pb_at = sl + STRIP;         /* strip B's scores of column j - 1 */
            ResidueWords tw;
            tw.start(tseq, cols);
            for (int j0 = 0; j0 <= wmax; j0 += 4, in_at += 4 * 32, out_at += 4 * 32) {
                if (CKPT && j0 > 0 && j0 % p16_ck(ALG) == 0) {
                    /* the state before iteration j0 */
                    uint4 *d = ckc + ((size_t)pass * p16_ck_blocks(ALG, wmax) + j0 / p16_ck(ALG) - 1) * P16_CK_U4 * 32;
#pragma unroll
                    for (int x = 0; x < P16_R / 4; ++x) {
                        d[x * 32] = make_uint4(H[4 * x], H[4 * x + 1], H[4 * x + 2], H[4 * x + 3]);
                        d[(x + P16_R / 4) * 32] = make_uint4(E[4 * x], E[4 * x + 1], E[4 * x + 2], E[4 * x + 3]);
                    }
                    d[P16_R / 2 * 32] = make_uint4(prev_f, dg, 0u, 0u);
                }
                uint32_t codes = tw.next(j0);
                if ((codes | (codes + big4)) & 0x80808080u) {
                    /* codes outside the alphabet read as letter 0 */
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (((codes >> (8 * b)) & 0xffu) >= (uint32_t)L) {
                            codes &= ~(0xffu << (8 * b));
                            status |= PB_ST_BADCODE;
                        }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + u;
                    const uint32_t v = top ? vtop : v_n[u];
                    vtop = __vadd2(vtop, top_step);
                    v_n[u] = j + 4 < rd ? __ldcg(in_at + u * 32) : vnone;
                    uint32_t hu = p16_prmt(v, prev_h, 0x5410u);      /* lo <- the row above */
                    uint32_t fu = p16_prmt(v, prev_f, 0x5432u);
                    const int8_t *pa_at = sl + ((codes >> (8 * u)) & 0xffu) * LETTER;
                    const uint4 pa4 = *reinterpret_cast<const uint4 *>(pa_at);
                    const uint4 pb4 = *reinterpret_cast<const uint4 *>(pb_at);
                    pb_at = pa_at + STRIP;
                    uint32_t hd = dg;
                    dg = hu;
                    uint32_t cmax = p16_splat(-bias);
                    uint32_t aop = 0u;               /* BIAS: the previous row's max(H_diag + s, E) - open */
#pragma unroll
                    for (int r = 0; r < P16_R; ++r) {
                        const uint32_t wa = r < 4 ? pa4.x : r < 8 ? pa4.y : r < 12 ? pa4.z : pa4.w;
                        const uint32_t wb = r < 4 ? pb4.x : r < 8 ? pb4.y : r < 12 ? pb4.z : pb4.w;
                        uint32_t sc;
                        switch (r & 3) {
                            case 0: sc = p16_pair<0>(wa, wb); break;
                            case 1: sc = p16_pair<1>(wa, wb); break;
                            case 2: sc = p16_pair<2>(wa, wb); break;
                            default: sc = p16_pair<3>(wa, wb); break;
                        }
                        uint32_t e, f, hn;           /* hn: H, or H - open */
                        if (BIAS) {
                            e = __viaddmax_s16x2(E[r], gE, H[r]);
                            const uint32_t a = ALG == PB_SW ? __viaddmax_s16x2_relu(hd, sc, e) : __viaddmax_s16x2(hd, sc, e);
                            const uint32_t ao = __vadd2(a, gO);
                            f = __viaddmax_s16x2(fu, gE, r == 0 ? hu : aop);
                            hn = __viaddmax_s16x2(f, gO, ao);
                            aop = ao;
                        } else {
                            e = __viaddmax_s16x2(E[r], gE, __vadd2(H[r], gO));
                            f = __viaddmax_s16x2(hu, gO, __vadd2(fu, gE));
                            hn = __vmaxs2(ALG == PB_SW ? __viaddmax_s16x2_relu(hd, sc, e)
                                                       : __viaddmax_s16x2(hd, sc, e), f);
                        }
                        E[r] = e;
                        hd = H[r];
                        H[r] = hn;
                        hu = hn;
                        fu = f;
                        if (ENDS && ALG == PB_SW && (r & 1)) cmax = __vimax3_s16x2(cmax, H[r - 1], hn);
                    }
                    if (more) out_at[u * 32] = p16_prmt(hu, fu, 0x7632u);     /* column j - 1 */
                    prev_h = hu;
                    prev_f = fu;
                    if (u == 0 && j0 == 0) {
                        /* the high half computed column -1: restore strip B's
                         * left boundary (H(i,-1), E = -inf) */
#pragma unroll
                        for (int r = 0; r < P16_R; ++r) {
                            const int lb2 = p16_left(ALG, sgf, r0 + P16_R + r, open, gap) - bias;
                            H[r] = (H[r] & 0xffffu) | ((uint32_t)(uint16_t)lb2 << 16);
                            E[r] = (E[r] & 0xffffu) | (NEG & 0xffff0000u);
                        }
                    }
                    if (ENDS && ALG == PB_SW && __vmaxs2(sbest, cmax) != sbest) {
                        /* past its half's bound: the column kept whole (the
                         * smallest row is looked up once per pass); columns
                         * outside the target only raise the bound */
                        const int c_lo = p16_lo(cmax), c_hi = p16_hi(cmax);
                        int ba = p16_lo(sbest), bb = p16_hi(sbest);
                        const bool up_a = c_lo > ba, up_b = c_hi > bb && j >= 1;
                        if (up_a) {
                            ba = c_lo;
                            if (j < cols) {
#pragma unroll
                                for (int x = 0; x < P16_R / 4; ++x)
                                    save[x] = make_uint4(H[4 * x], H[4 * x + 1], H[4 * x + 2], H[4 * x + 3]);
                                sa.score = c_lo + bias; sa.j = j;
                                bb = max(bb, c_lo - 1);
                            }
                        }
                        if (up_b) {
                            bb = max(bb, c_hi);
                            if (j <= cols) {
#pragma unroll
                                for (int x = 0; x < P16_R / 4; ++x)
                                    save[P16_R / 4 + x] = make_uint4(H[4 * x], H[4 * x + 1], H[4 * x + 2], H[4 * x + 3]);
                                sb.score = c_hi + bias; sb.j = j - 1;
                                ba = max(ba, c_hi - 1);
                            }
                        }
                        sbest = (uint32_t)(uint16_t)ba | ((uint32_t)(uint16_t)bb << 16);
                    }
                    if (ENDS && ALG != PB_SW) {
                        /* last column (strip A at j = cols - 1, strip B one
                         * iteration later): SG's last-column maximum over rows
                         * below rows - 1 (smallest row on ties), and the corner */
                        if ((unsigned)(j - (cols - 1)) <= 1u && (ALG == PB_SG || lastpass)) {
                            const int hsel = j == cols - 1 ? 0 : 1;
                            const int ib = r0 + hsel * P16_R;
#pragma unroll
                            for (int r = 0; r < P16_R; ++r) {
                                const int hv = (hsel ? p16_hi(H[r]) : p16_lo(H[r])) + bias;
                                const int i = ib + r;
                                if (ALG == PB_SG && (sgf & PB_S1_END) && i < ilast && hv > lc_h) { lc_h = hv; lc_i = i; }
                                if (i == ilast) corner = hv;
                            }
                        }
                        if (ALG == PB_SG && (sgf & PB_S2_END) && lastpass) {
                            const int jj = j - half_last;
                            uint32_t lastv = 0u;
#pragma unroll
                            for (int r = 0; r < P16_R; ++r) if (r == r_last) lastv = H[r];
                            const int hv = (half_last ? p16_hi(lastv) : p16_lo(lastv)) + bias;
                            if (jj >= 0 && jj < cols && hv > lr_h) { lr_h = hv; lr_j = jj; }
                        }
                    }
                }
            }
            if (ENDS && ALG == PB_SW) {
                if (sa.j >= 0) {
                    int rr = P16_R - 1;
#pragma unroll
                    for (int x = P16_R / 4 - 1; x >= 0; --x) {
                        const uint4 w = save[x];
                        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int y = 3; y >= 0; --y) if (p16_lo(ws[y]) == sa.score - bias) rr = 4 * x + y;
                    }
                    sa.i = r0 + rr;
                }
                if (sb.j >= 0) {
                    int rr = P16_R - 1;
#pragma unroll
                    for (int x = P16_R / 4 - 1; x >= 0; --x) {
                        const uint4 w = save[P16_R / 4 + x];
                        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int y = 3; y >= 0; --y) if (p16_hi(ws[y]) == sb.score - bias) rr = 4 * x + y;
                    }
                    sb.i = r0 + P16_R + rr;
                }
                const P16Best cand[2] = {sa, sb};
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const P16Best c = cand[x];
                    if (c.j >= 0 && (c.score > best.score || (c.score == best.score && c.j < best.j))) best = c;
                }
            }
        }
        if (valid) {
            pb_pair_out o;
            if (ENDS) {
                int sc, eq, er;
                if (ALG == PB_SW) {
                    sc = best.score; eq = best.i; er = best.j;
                } else if (ALG == PB_NW) {
                    sc = corner; eq = ilast; er = cols - 1;
                } else {
                    /* src/sg.c:160-242 */
                    const bool s1e = sgf & PB_S1_END, s2e = sgf & PB_S2_END;
                    sc = INT_MIN; eq = rows; er = cols;
                    if (s1e && lc_i >= 0) { sc = lc_h; eq = lc_i; er = cols - 1; }
                    if (s1e && s2e) {
                        if (lr_h > sc || (lr_h == sc && lr_j < er)) { sc = lr_h; eq = ilast; er = lr_j; }
                    } else if (s2e) {
                        if (lr_h > sc) { sc = lr_h; eq = ilast; er = lr_j; }
                    }
                    if ((s1e && corner > sc) || (!s1e && !s2e)) { sc = corner; eq = ilast; er = cols - 1; }
                }
                o.score = sc; o.end_query = eq; o.end_ref = er;
                o.max_h = ALG == PB_SW ? sc : bd.ub;
            } else {
                o.score = 0; o.end_query = 0; o.end_ref = 0;
                o.max_h = bd.ub;
            }
            o.matches = o.similar = o.length = 0;
            /* the width verdicts read sound bounds (see p16_check) */
            o.min_h_real = bd.lb;
            o.min_f_real = bd.lb - open;
            o.max_stat_real = ((rows + 31) & ~31) + cols;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                o.min_h_pad[x] = bd.lb;
                o.max_stat_pad[x] = o.max_stat_real;
                o.min_f_pad[x] = bd.lb - open;
            }
            o.status = status | PB_ST_BOUNDED;
            p.out[item] = o;
        }
    }
}

/*
 * The traceback of one task's items, a lane each: from its end cell back
 * along the path the reference's tie rules select. A lane restarts the
 * dynamic program at the checkpoint before its cell -- the column state at
 * the start of the cell's block of p16_ck columns, the bottom row of the
 * pass above -- and recomputes the block up to the cell with the direction
 * bits of its 32 rows in shared memory, walks until it leaves the block, and
 * goes on with the next one. The lanes of a warp run their blocks in step,
 * each its own pass and columns, so a task takes as many blocks as its
 * longest path: two per pass for a global alignment, a handful for the local
 * alignment of unrelated sequences, where direction bits had to be computed
 * and stored for the whole prefix before the end cell. All against all, 524 k
 * protein pairs: 158 ms of prefix pass and walk -> 7.5 ms; 1 M reads, NW: 3.2
 * ms of walk over stored bits -> 7.0 ms, against 19 ms less in the forward
 * pass. Bound by the ALU and FMA pipes for DNA (58% each), by latency for
 * proteins, whose scores leave room for four warps an SM.
 *
 * The bits (the four decisions of the file comment) are signs of differences;
 * of two rows, one permute spreads the signs over four bytes (strips A and B
 * of the even row, then of the odd one) of which a mask keeps bit r / 2: 8 ALU
 * and 8 FMA operations per row of two cells.
 *
 * MODE 0: matches, similar and length into out[item]; 1 (FASTSTATS in one
 * pass): the whole prefix output into out2[item], the bounds being those of
 * the prefix up to the end cell; 2: the path's steps, written backwards from
 * the end of the item's op buffer -- 0 a diagonal step (query and target
 * residue aligned), 1 a step up a vertical gap (a query residue against a
 * gap), 2 a step left along a horizontal gap (a target residue against a
 * gap) -- with the cell where the walk stopped. The decisions are those the
 * reference's trace tables hold (src/sw_trace.c:138-147: DIAG when H ==
 * H_diag, else DEL when H == F, else INS; DIAG_F / DIAG_E when the gap opened
 * by strict >), followed as its CIGAR builder does (src/cigar_template.c:
 * 143-243).
 */
template <int ALG, int MODE, bool BIAS>
__global__ void __launch_bounds__(P16_TR_WARPS * 32, 7)
k_p16_trace(pb_job job, P16Params p, const int *__restrict__ tlist, int ntl, const pb_pair_out *__restrict__ ends,
            int *counter)
{
    extern __shared__ __align__(16) int8_t s_mem[];
    constexpr int LETTER = 1024, STRIP = 512, CK = p16_ck(ALG);
    const int L = p.nletters;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int open = p.open, gap = p.gap, sgf = p.sgflags;
    const int bias = BIAS ? open : 0;
    /* shared memory: [matrix L x L int8, padded to 16] then per warp [bits of
     * a block][scores] */
    const int mat_bytes = p.mat8 ? ((L * L + 15) & ~15) : 0;
    int8_t *s_mat = s_mem;
    int8_t *wmem = s_mem + mat_bytes + (size_t)wid * (CK * 512 + L * LETTER);
    uint4 *tile = reinterpret_cast<uint4 *>(wmem) + lane;
    int8_t *sl = wmem + CK * 512 + lane * 16;
    if (p.mat8)
        for (int x = threadIdx.x; x < L * L; x += blockDim.x) s_mat[x] = (int8_t)(p.mat8[x] + bias);
    __syncthreads();
    const uint32_t gO = p16_splat(-open), gE = p16_splat(-gap);
    const uint32_t b4 = 0x01010101u * (uint32_t)(uint8_t)bias;

    for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(counter, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= ntl) break;
        const int task = tlist[k];
        const int s = task * 32 + lane;
        const bool valid = s < p.nitems && p.order[s] >= 0;
        const int item = valid ? p.order[s] : 0;
        const int rows = valid ? p.rows[item] : 0, cols = valid ? p.cols[item] : 0;
        const int wmax = p.task_wmax[task], npass = p.task_npass[task];
        const int stride = p16_cols(wmax);
        const uint32_t *ckr = reinterpret_cast<const uint32_t *>(p.ckpt + p.task_ckpt[task]) + lane;
        const uint4 *ckc = p.ckpt + p.task_ckpt[task] + p16_ck_col(ALG, npass, wmax, 0, 0) + lane;
        const int ti = p.nt ? item % p.nt : item;
        const uint8_t *tseq = p.targets + (valid ? p.toff[ti] : 0);
        const uint8_t *qseq = nullptr;
        const int8_t *prof8 = nullptr;
        int lp = 0;
        if (p.mat8) {
            qseq = p.qall + (valid ? p.qoff[item] : 0);
        } else {
            const ProfDesc pd = p.profs[p.nt ? item / p.nt : 0];
            qseq = pd.qcodes;
            prof8 = pd.prof8;
            lp = pd.lp;
        }
        pb_pair_out e;
        if (valid) e = ends[item];
        else memset(&e, 0, sizeof e);
        int i = e.end_query, j = e.end_ref, v = e.score;
        /* an end outside the computed region (a FASTSTATS item whose prefix
         * pass was not needed): nothing to walk */
        bool active = valid && i >= 0 && j >= 0 && i < rows && j < cols;
        bool need2 = true;
        if (MODE == 1 && valid) {
            need2 = pb_needs_pass2(&job, &e) != 0;
            active = active && need2;
        }
        const P16Bounds bd = p16_bounds(ALG, rows, cols, open, gap, p.mmax, p.mmin);
        const int negv = bd.lb - open - 1;
        const uint32_t NEG = p16_splat(negv);
        const int cap = rows + cols;
        uint8_t *ops = MODE == 2 && valid ? p.ops + p.ops_off[item] : nullptr;
        const bool started = active;
        int M = 0, S = 0, n = 0, state = 0;                  /* state: 0 H, 1 F, 2 E */
        int staged = -1;
        if (ALG == PB_SW && v <= 0) active = false;
        while (__any_sync(0xffffffffu, active)) {
            const int pass = active ? i >> 5 : 0, r0 = pass * P16_PASS;
            const int jt = active ? j + ((i >> 4) & 1) : 0;  /* the iteration of the cell */
            const int jb = jt / CK * CK;
            /* the scores (BIAS: + open) of this pass's rows */
            if (active && pass != staged) {
                staged = pass;
                if (p.mat8) {
                    uint32_t qc[8];
#pragma unroll
                    for (int w = 0; w < 8; ++w) {
                        uint32_t word = 0;
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            const int x = r0 + 4 * w + b;
                            uint32_t c = 255u;
                            if (x < rows) {
                                c = qseq[x];
                                if (c >= (uint32_t)L) c = 0;
                            }
                            word |= c << (8 * b);
                        }
                        qc[w] = word;
                    }
                    for (int a = 0; a < L; ++a) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t word[4];
#pragma unroll
                            for (int w = 0; w < 4; ++w) {
                                word[w] = 0;
#pragma unroll
                                for (int b = 0; b < 4; ++b) {
                                    const uint32_t c = (qc[4 * h + w] >> (8 * b)) & 0xffu;
                                    const uint32_t x = c == 255u ? (uint32_t)(uint8_t)bias
                                                                 : (uint32_t)(uint8_t)s_mat[a * L + c];
                                    word[w] |= x << (8 * b);
                                }
                            }
                            *reinterpret_cast<uint4 *>(sl + a * LETTER + h * STRIP) =
                                make_uint4(word[0], word[1], word[2], word[3]);
                        }
                    }
                } else {
                    const bool in = r0 + P16_PASS <= lp;
                    for (int a = 0; a < L; ++a) {
                        const int4 *src = reinterpret_cast<const int4 *>(prof8 + (size_t)a * lp + (in ? r0 : 0));
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            int4 x = in ? src[h] : make_int4(0, 0, 0, 0);
                            if (BIAS) {
                                x.x = (int)__vadd4((uint32_t)x.x, b4); x.y = (int)__vadd4((uint32_t)x.y, b4);
                                x.z = (int)__vadd4((uint32_t)x.z, b4); x.w = (int)__vadd4((uint32_t)x.w, b4);
                            }
                            *reinterpret_cast<int4 *>(sl + a * LETTER + h * STRIP) = x;
                        }
                    }
                }
            }
            /* the state before iteration jb */
            uint32_t H[P16_R], E[P16_R], dg, prev_h, prev_f;
            if (jb == 0) {
#pragma unroll
                for (int r = 0; r < P16_R; ++r) {
                    const int la = p16_left(ALG, sgf, r0 + r, open, gap) - bias;
                    const int lb2 = p16_left(ALG, sgf, r0 + P16_R + r, open, gap) - bias;
                    H[r] = (uint32_t)(uint16_t)la | ((uint32_t)(uint16_t)lb2 << 16);
                    E[r] = NEG;
                }
                dg = (uint32_t)(uint16_t)(p16_left(ALG, sgf, r0 - 1, open, gap) - bias);
                prev_h = (uint32_t)(uint16_t)(p16_left(ALG, sgf, r0 + P16_R - 1, open, gap) - bias);
                prev_f = NEG & 0xffffu;
            } else {
                const uint4 *d = ckc + ((size_t)pass * p16_ck_blocks(ALG, wmax) + jb / CK - 1) * P16_CK_U4 * 32;
#pragma unroll
                for (int x = 0; x < P16_R / 4; ++x) {
                    const uint4 h4 = __ldcg(d + x * 32), e4 = __ldcg(d + (x + P16_R / 4) * 32);
                    H[4 * x] = h4.x; H[4 * x + 1] = h4.y; H[4 * x + 2] = h4.z; H[4 * x + 3] = h4.w;
                    E[4 * x] = e4.x; E[4 * x + 1] = e4.y; E[4 * x + 2] = e4.z; E[4 * x + 3] = e4.w;
                }
                const uint4 m4 = __ldcg(d + P16_R / 2 * 32);
                prev_f = m4.x;
                dg = m4.y;
                prev_h = H[P16_R - 1];
            }
            /* the row above: row -1 (as the forward kernel steps it), or the
             * pass above's bottom row */
            const bool top = pass == 0;
            const int tstep = (ALG == PB_SW || (ALG == PB_SG && (sgf & PB_S2_BEG))) ? 0 : gap;
            uint32_t vtop = p16_prmt((uint32_t)(uint16_t)(p16_top(ALG, sgf, 0, open, gap) - bias - jb * tstep), NEG, 0x5410u);
            const uint32_t top_step = (uint32_t)(uint16_t)(-tstep);
            const uint32_t *in_row = ckr + (top ? 0 : p16_ck_row(wmax, pass - 1, 0)) + 32;
            const int rd = top ? 0 : wmax;
            const uint32_t vnone = p16_prmt(0u, NEG, 0x5410u);
            uint32_t v_n[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) v_n[x] = jb + x < rd ? __ldcg(in_row + (size_t)(jb + x) * 32) : vnone;
            ResidueWords tw;
            tw.start(tseq + jb, active ? cols - jb : 0);
            int cb = active && jb > 0 ? tseq[jb - 1] : 0;
            if (cb >= L) cb = 0;
            const int8_t *pb_at = sl + cb * LETTER + STRIP;
            const int cnt = __reduce_max_sync(0xffffffffu, active ? jt - jb + 1 : 0);
            for (int x0 = 0; x0 < cnt; x0 += 4) {
                uint32_t codes = tw.next(x0);
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (((codes >> (8 * b)) & 0xffu) >= (uint32_t)L) codes &= ~(0xffu << (8 * b));
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int x = x0 + u, jj = jb + x;
                    const uint32_t vv = top ? vtop : v_n[u];
                    vtop = __vadd2(vtop, top_step);
                    v_n[u] = jj + 4 < rd ? __ldcg(in_row + (size_t)(jj + 4) * 32) : vnone;
                    uint32_t hu = p16_prmt(vv, prev_h, 0x5410u);
                    uint32_t fu = p16_prmt(vv, prev_f, 0x5432u);
                    const int8_t *pa_at = sl + ((codes >> (8 * u)) & 0xffu) * LETTER;
                    const uint4 pa4 = *reinterpret_cast<const uint4 *>(pa_at);
                    const uint4 pb4 = *reinterpret_cast<const uint4 *>(pb_at);
                    pb_at = pa_at + STRIP;
                    uint32_t hd = dg;
                    dg = hu;
                    uint32_t aD = 0u, aF = 0u, aE = 0u, aV = 0u;
                    uint32_t dD = 0u, dF = 0u, dE = 0u, dV = 0u;
#pragma unroll
                    for (int r = 0; r < P16_R; ++r) {
                        const uint32_t wa = r < 4 ? pa4.x : r < 8 ? pa4.y : r < 12 ? pa4.z : pa4.w;
                        const uint32_t wb = r < 4 ? pb4.x : r < 8 ? pb4.y : r < 12 ? pb4.z : pb4.w;
                        uint32_t sc;
                        switch (r & 3) {
                            case 0: sc = p16_pair<0>(wa, wb); break;
                            case 1: sc = p16_pair<1>(wa, wb); break;
                            case 2: sc = p16_pair<2>(wa, wb); break;
                            default: sc = p16_pair<3>(wa, wb); break;
                        }
                        const uint32_t ho = BIAS ? H[r] : __vadd2(H[r], gO);
                        const uint32_t fo = BIAS ? hu : __vadd2(hu, gO);
                        const uint32_t ee = __vadd2(E[r], gE), fe = __vadd2(fu, gE);
                        const uint32_t en = __vmaxs2(ho, ee), fn = __vmaxs2(fo, fe);
                        const uint32_t hdg = __vadd2(hd, sc);
                        const uint32_t h = ALG == PB_SW ? __vimax3_s16x2_relu(hdg, en, fn) : __vimax3_s16x2(hdg, en, fn);
                        const uint32_t hn = BIAS ? __vadd2(h, gO) : h;
                        const uint32_t nD = __vsub2(hdg, h), nF = __vsub2(fn, h);
                        const uint32_t nE = __vsub2(ee, ho), nV = __vsub2(fe, fo);
                        if (r & 1) {
                            const uint32_t m = 0x01010101u << (r >> 1);
                            aD |= p16_prmt(dD, nD, 0xfdb9u) & m;
                            aF |= p16_prmt(dF, nF, 0xfdb9u) & m;
                            aE |= p16_prmt(dE, nE, 0xfdb9u) & m;
                            aV |= p16_prmt(dV, nV, 0xfdb9u) & m;
                        }
                        dD = nD; dF = nF; dE = nE; dV = nV;
                        E[r] = en;
                        hd = H[r];
                        H[r] = hn;
                        hu = hn;
                        fu = fn;
                    }
                    tile[x * 32] = make_uint4(aD, aF, aE, aV);
                    prev_h = hu;
                    prev_f = fu;
                    if (u == 0 && jj == 0) {
                        /* the high half computed column -1 */
#pragma unroll
                        for (int r = 0; r < P16_R; ++r) {
                            const int lb2 = p16_left(ALG, sgf, r0 + P16_R + r, open, gap) - bias;
                            H[r] = (H[r] & 0xffffu) | ((uint32_t)(uint16_t)lb2 << 16);
                            E[r] = (E[r] & 0xffffu) | (NEG & 0xffff0000u);
                        }
                    }
                }
            }
            /* the walk inside the block (each step moves up or left or changes
             * from H to a gap, so it ends) */
            while (active) {
                const int half = (i >> 4) & 1, x = j + half - jb;
                if ((i >> 5) != pass || x < 0) break;
                const int bit = p16_bit(i);
                const uint4 w = tile[x * 32];
                if (state == 0) {
                    if (!((w.x >> bit) & 1u)) {
                        int qc = qseq[i], tc = tseq[j];
                        if (qc >= L) qc = 0;
                        if (tc >= L) tc = 0;
                        /* the staged score of this cell */
                        const int sc = (int)sl[tc * LETTER + half * STRIP + (i & 15)] - bias;
                        M += qc == tc;
                        S += sc > 0;
                        v -= sc;
                        if (MODE == 2 && n < cap) ops[cap - 1 - n] = 0;
                        ++n;
                        --i;
                        --j;
                    } else {
                        state = ((w.y >> bit) & 1u) ? 2 : 1;
                    }
                } else if (state == 1) {
                    if (MODE == 2 && n < cap) ops[cap - 1 - n] = 1;
                    ++n;
                    if ((w.w >> bit) & 1u) { v += open; state = 0; } else { v += gap; }
                    --i;
                } else {
                    if (MODE == 2 && n < cap) ops[cap - 1 - n] = 2;
                    ++n;
                    if ((w.z >> bit) & 1u) { v += open; state = 0; } else { v += gap; }
                    --j;
                }
                if (i < 0 || j < 0 || (ALG == PB_SW && state == 0 && v <= 0) || n >= cap) active = false;
            }
            __syncwarp();
        }
        if (!valid) continue;
        if (MODE == 2) {
            int *info = p.path_info + 3 * (size_t)item;
            info[0] = started ? n : -1; info[1] = i; info[2] = j;
        } else if (MODE == 0) {
            pb_pair_out *o = p.out + item;
            o->matches = M; o->similar = S; o->length = n;
        } else {
            /* as the prefix pass (ENDS off) writes it */
            const int pr = need2 ? e.end_query + 1 : 1, pc = need2 ? e.end_ref + 1 : 1;
            const P16Bounds b2 = p16_bounds(ALG, pr, pc, open, gap, p.mmax, p.mmin);
            pb_pair_out o;
            o.score = 0; o.end_query = 0; o.end_ref = 0;
            o.max_h = b2.ub;
            o.matches = M; o.similar = S; o.length = n;
            o.min_h_real = b2.lb;
            o.min_f_real = b2.lb - open;
            o.max_stat_real = ((pr + 31) & ~31) + pc;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                o.min_h_pad[x] = b2.lb;
                o.max_stat_pad[x] = o.max_stat_real;
                o.min_f_pad[x] = b2.lb - open;
            }
            o.status = e.status | PB_ST_BOUNDED;
            p.out2[item] = o;
        }
    }
}

/* per item: rows, columns, eligibility and the sort key (eligible first,
 * then by query group, passes and columns, all descending) */
__global__ void k_p16_setup(P16Setup q, int *__restrict__ rows, int *__restrict__ cols,
                            unsigned long long *__restrict__ keys, int *__restrict__ idx,
                            int *__restrict__ counts)
{
    const int item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= q.nitems) return;
    const int ti = q.nt ? item % q.nt : item;
    int r = q.qlim ? q.qlim[item] : (q.qlen ? q.qlen[item] : q.prof_qlen[item / q.nt]);
    const int c = q.tlim ? q.tlim[item] : q.tlen[ti];
    rows[item] = r;
    cols[item] = c;
    idx[item] = item;
    bool ok = r >= 1 && c >= 1 && c <= q.max_cols && r <= 65535 && !((q.intra_mask >> p16_bucket(r, c)) & 1u);
    if (ok) {
        const P16Bounds b = p16_bounds(q.alg, r, c, q.open, q.gap, q.mmax, q.mmin);
        ok = p16_fits(b, q.open, q.gap);
    }
    if (ok) {
        const unsigned long long grp = q.group ? (unsigned long long)(q.group[item] & 0xfffff)
                                               : (q.nt ? (unsigned long long)(item / q.nt) & 0xfffff : 0ull);
        const unsigned long long np = (unsigned long long)((r + 31) / 32) & 0x7ff;
        keys[item] = (1ull << 63) | (grp << 43) | (np << 32) | ((unsigned long long)c & 0xffffffffull);
        atomicAdd(&counts[0], 1);
    } else {
        keys[item] = 0ull;
    }
}

/* per task (a warp each): widest target, passes, shared query, uint4s of its
 * checkpoints */
__global__ void k_p16_tasks(P16Params p, int ntasks, const int *__restrict__ group, int *__restrict__ twmax,
                            int *__restrict__ tnpass, int *__restrict__ tshared, long long *__restrict__ tckpt,
                            int ckpt)
{
    const int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (task >= ntasks) return;
    const int s = task * 32 + lane;
    const bool valid = s < p.nitems && p.order[s] >= 0;
    const int item = valid ? p.order[s] : -1;
    int c = valid ? p.cols[item] : 0, r = valid ? p.rows[item] : 0;
    long long src = -1;
    if (valid) {
        if (p.mat8) src = group ? (long long)group[item] : -2 - (long long)item;   /* pairs: one query per item */
        else src = p.nt ? item / p.nt : 0;
    }
    long long src0 = __shfl_sync(0xffffffffu, src, 0);
    const bool same = __all_sync(0xffffffffu, !valid || src == src0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c = max(c, __shfl_xor_sync(0xffffffffu, c, o));
        r = max(r, __shfl_xor_sync(0xffffffffu, r, o));
    }
    if (lane == 0) {
        const int np = (r + P16_PASS - 1) / P16_PASS;
        twmax[task] = c;
        tnpass[task] = np;
        tshared[task] = p.mat8 ? (same && group != nullptr) : 1;
        tckpt[task] = ckpt ? (long long)p16_ck_col(p.alg, np, c, np, 0) : 0;
    }
}

}  // namespace pb

namespace pb {

/* Is the record pb_chain_resolve builds from an item's bounded extremes
 * (pb_pair_out with PB_ST_BOUNDED: max_h an upper bound except in SW, where
 * it is the score; minima lower bounds; statistics maxima upper bounds) the
 * one it would build from exact extremes? Each width the chain visits must
 * either be CLEAN by the bounds (sound: the bounds contain the exact
 * values), be SAT by a value the item is known to reach (the score is a
 * visited H: above POS_LIMIT, or in a scan kernel below NEG_LIMIT), or be
 * decided by the lane-exact kernel, which does not read the extremes. */
__device__ bool p16_definite(const pb_job &job, const pb_pair_out &o, int qlen, int tlen)
{
    const pb_mode *m = &job.mode;
    if (job.bits < 0) return true;                         /* serial forms: exact values only */
    if (pb_job_is_faststats(&job)) return true;            /* score pass exact; prefix pass CLEAN or lane-exact */
    if (m->alg == PB_SW && !m->stats) return true;         /* SW score-only reads max_h = score only */
    const int w3[3] = {8, 16, 32};
    int f, l;
    pb_job_widths(&job, &f, &l);
    for (int t = f; t <= l; ++t) {
        const int w = w3[t];
        const int v = pb_resolve_tier(m, w, &o, qlen, tlen);
        if (pb_lane_applies(m, w) && (v != PB_CLEAN || pb_lane_forced(m, w))) continue;
        if (v == PB_CLEAN) return true;
        if (v != PB_SAT) return false;
        const int64_t imin = int_min_w(w), imax = int_max_w(w);
        const int64_t neg = ((-(int64_t)m->open < m->mmin) ? imin + m->open : imin - m->mmin) + 1;
        const int64_t pos = imax - m->mmax - 1;
        const int L = lanes_of(w);
        const int64_t padlen = ((int64_t)qlen + L - 1) / L * L;
        bool proven = (int64_t)o.score > pos;
        if (!m->striped && (int64_t)o.score < neg) proven = true;
        if (m->alg != PB_SW && m->striped && !m->stats && boundary_h(m, (int)padlen - 1, 0) - m->open < neg)
            proven = true;
        if (!proven) return false;
    }
    return true;
}

__global__ void k_p16_check(pb_job job, P16Params p, int *__restrict__ rest, int *__restrict__ nrest)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.nitems) return;
    const int item = p.order[s];
    if (item < 0) return;
    if (!p16_definite(job, p.out[item], p.rows[item], p.cols[item])) rest[atomicAdd(nrest, 1)] = item;
}

/* Task alignment to query groups: the eligible items sorted by (group,
 * passes, columns) are laid out so that every group starts a task (each
 * group padded with -1 entries to a multiple of 32). No task then mixes two
 * queries, and every task of a grouped batch takes the shared-query
 * variant. */
__global__ void k_pad_heads(const unsigned long long *__restrict__ keys, int n, int *__restrict__ head)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) head[s] = s == 0 || ((keys[s] >> 43) & 0xfffffull) != ((keys[s - 1] >> 43) & 0xfffffull);
}

__global__ void k_pad_counts(const int *__restrict__ gstart, int ng, int n, int *__restrict__ pcount)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < ng) pcount[g] = ((g + 1 < ng ? gstart[g + 1] : n) - gstart[g] + 31) & ~31;
}

__global__ void k_pad_scatter(const int *__restrict__ order, int n, const int *__restrict__ gid,
                              const int *__restrict__ gstart, const int *__restrict__ pstart, int *__restrict__ out)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) {
        const int g = gid[s] - 1;
        out[pstart[g] + (s - gstart[g])] = order[s];
    }
}

__global__ void k_mat_to_int8(const int32_t *__restrict__ m, int n, int8_t *__restrict__ m8)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) m8[k] = (int8_t)m[k];
}

__global__ void k_iota_int(int *__restrict__ v, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) v[k] = k;
}

__global__ void k_copy_int(const int *__restrict__ src, int n, int *__restrict__ dst)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[k] = src[k];
}

struct P16Frees {
    cudaStream_t st;
    std::vector<void *> v;
    explicit P16Frees(cudaStream_t s) : st(s) {}
    template <typename T> T *add(T *q) { if (q) v.push_back((void *)q); return q; }
    ~P16Frees() { for (void *q : v) cudaFreeAsync(q, st); }
};

namespace {

#define PB_P16(call)                                           \
    do {                                                       \
        if ((call) != cudaSuccess) {                           \
            fprintf(stderr, "pb_pair16: %s failed\n", #call);  \
            return -1;                                         \
        }                                                      \
    } while (0)

int p16_warps(bool shared, int L) { return shared || L <= 8 ? 8 : 4; }

size_t p16_smem(bool shared, int L, bool mat)
{
    const size_t mat_bytes = mat ? ((size_t)(L * L + 15) & ~(size_t)15) : 0;
    const size_t warp_bytes = (size_t)L * (shared ? P16_ROW : 32 * P16_PASS);
    return mat_bytes + warp_bytes * p16_warps(shared, L);
}

typedef void (*p16_kernel_t)(P16Params, const int *, int, int *);

template <int ALG, bool CKPT, bool ENDS, bool BIAS>
p16_kernel_t pick3(bool shared, int warps)
{
    if (shared) return k_p16<ALG, CKPT, ENDS, true, 8, BIAS>;
    return warps == 8 ? k_p16<ALG, CKPT, ENDS, false, 8, BIAS> : k_p16<ALG, CKPT, ENDS, false, 4, BIAS>;
}

template <bool BIAS>
p16_kernel_t pick(int alg, bool ckpt, bool ends, bool shared, int warps)
{
    if (alg == PB_SW) {
        if (!ends) return pick3<PB_SW, true, false, BIAS>(shared, warps);
        return ckpt ? pick3<PB_SW, true, true, BIAS>(shared, warps) : pick3<PB_SW, false, true, BIAS>(shared, warps);
    }
    if (alg == PB_NW)
        return ckpt ? pick3<PB_NW, true, true, BIAS>(shared, warps) : pick3<PB_NW, false, true, BIAS>(shared, warps);
    return ckpt ? pick3<PB_SG, true, true, BIAS>(shared, warps) : pick3<PB_SG, false, true, BIAS>(shared, warps);
}

/* the current device's memory in bytes */
size_t device_memory()
{
    static std::mutex mu;
    static std::vector<size_t> seen;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if ((size_t)dev >= seen.size()) seen.resize(dev + 1, 0);
    if (!seen[dev]) {
        size_t free_b = 0, total = 0;
        seen[dev] = cudaMemGetInfo(&free_b, &total) == cudaSuccess && total ? total : (size_t)24 << 30;
    }
    return seen[dev];
}

/* The chunks that ntasks tasks with `all` bytes of checkpoints run in: chunks
 * of at most a third of the device's memory, so that one of the largest tasks
 * (about 20 MB each at 1500 x 1500) still fills the SMs, but not so large that
 * the pool grows by more than half of what is free, which other allocators and
 * processes may need. The free memory is asked for only where the pool would
 * have to grow (by more than an eighth of what it holds unused): on a shared
 * host that call takes 0.1 to 90 ms, at random (18.9 ms passes of 1 M reads
 * became 20-110 ms). */
size_t p16_chunks(size_t ntasks, size_t all)
{
    const size_t cap = device_memory() / 3;
    auto chunks = [&](size_t bytes) { return std::min(ntasks, all / std::max<size_t>(bytes, 1) + 1); };
    int dev = 0;
    cudaMemPool_t pool;
    uint64_t reserved = 0, used = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetMemPool(&pool, dev) == cudaSuccess) {
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved);
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used);
    }
    const size_t spare = reserved > used ? (size_t)(reserved - used) : 0, n = chunks(cap);
    if (all / n <= spare + spare / 8) return n;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) { cudaGetLastError(); return n; }
    return chunks(std::min(cap, std::max(spare, free_b / 2 + spare / 2)));
}

typedef void (*p16_trace_t)(pb_job, P16Params, const int *, int, const pb_pair_out *, int *);

template <bool BIAS>
p16_trace_t pick_trace(int alg, int mode)
{
    if (alg == PB_SW)
        return mode == 0 ? k_p16_trace<PB_SW, 0, BIAS> : mode == 1 ? k_p16_trace<PB_SW, 1, BIAS> : k_p16_trace<PB_SW, 2, BIAS>;
    if (alg == PB_NW) return mode == 2 ? k_p16_trace<PB_NW, 2, BIAS> : k_p16_trace<PB_NW, 0, BIAS>;
    return mode == 2 ? k_p16_trace<PB_SG, 2, BIAS> : k_p16_trace<PB_SG, 0, BIAS>;
}

}  // namespace

int p16_pass(const pb_job &job, const pb_batch *b, int prefix, const pb_pair_out *ends, pb_pair_out *out,
             const int *group, int *d_rest, int *n_rest, cudaStream_t st,
             uint8_t *d_ops, const int64_t *d_ops_off, int *d_path_info, unsigned intra_mask, pb_pair_out *out2)
{
    const pb_mode *m = &job.mode;
    const bool dbmode = b->nprofs > 0;
    const int N = dbmode ? b->npairs * b->nprofs : b->npairs;
    *n_rest = 0;
    if (N <= 0) return 0;
    if ((long long)(dbmode ? (long long)b->npairs * b->nprofs : b->npairs) > INT32_MAX) return -1;
    const bool paths = d_ops != nullptr;
    const bool walk = prefix || out2 || (m->stats && !pb_job_is_faststats(&job));
    const bool ckpt = walk || paths;
    const bool ends_on = !prefix;
    P16Frees frees(st);
    /* alphabet and score source; anything the kernels cannot take goes to the exact kernel */
    int L = 0, mmax = 0, mmin = 0;
    bool usable = true;
    int8_t *d_mat8 = nullptr;
    ProfDesc *d_profs = nullptr;
    int *d_pql = nullptr;
    if (dbmode) {
        L = b->profs[0]->size;
        mmax = b->profs[0]->mmax; mmin = b->profs[0]->mmin;
        std::vector<ProfDesc> h(b->nprofs);
        std::vector<int> ql(b->nprofs);
        for (int q = 0; q < b->nprofs; ++q) {
            const pb_device_profile *dp = b->profs[q];
            usable = usable && dp->fits8 && dp->size == L && dp->d_prof8;
            h[q].prof = dp->d_prof32; h[q].prof8 = dp->d_prof8; h[q].qcodes = dp->d_qcodes;
            h[q].qlen = dp->qlen; h[q].lp = dp->lp; h[q].size = dp->size; h[q].pad_ = 0;
            ql[q] = dp->qlen;
            mmax = dp->mmax > mmax ? dp->mmax : mmax;
            mmin = dp->mmin < mmin ? dp->mmin : mmin;
        }
        if (usable) {
            PB_P16(cudaMallocAsync((void **)&d_profs, sizeof(ProfDesc) * b->nprofs, st));
            frees.add(d_profs);
            PB_P16(cudaMallocAsync((void **)&d_pql, sizeof(int) * b->nprofs, st));
            frees.add(d_pql);
            PB_P16(cudaMemcpyAsync(d_profs, h.data(), sizeof(ProfDesc) * b->nprofs, cudaMemcpyHostToDevice, st));
            PB_P16(cudaMemcpyAsync(d_pql, ql.data(), sizeof(int) * b->nprofs, cudaMemcpyHostToDevice, st));
            PB_P16(cudaStreamSynchronize(st));      /* the host vectors die at return */
        }
    } else {
        L = b->msize; mmax = b->mmax; mmin = b->mmin;
        usable = b->d_mat && b->mmin >= -128 && b->mmax <= 127;
        if (usable) {
            PB_P16(cudaMallocAsync((void **)&d_mat8, (size_t)L * L, st));
            frees.add(d_mat8);
            k_mat_to_int8<<<(L * L + 255) / 256, 256, 0, st>>>(b->d_mat, L * L, d_mat8);
            pb_diag_count_launch(1);
        }
    }
    usable = usable && L >= 1 && L <= 32;
    if (!usable) {
        /* nothing for the pair kernels: every item to the exact kernel */
        k_iota_int<<<(N + 255) / 256, 256, 0, st>>>(d_rest, N);
        pb_diag_count_launch(1);
        *n_rest = N;
        PB_P16(cudaStreamSynchronize(st));
        return 0;
    }
    /* per item: rows, columns, eligibility, sort */
    int *rows = nullptr, *cols = nullptr, *idx = nullptr, *order = nullptr, *counts = nullptr;
    unsigned long long *keys = nullptr, *keys_sorted = nullptr;
    PB_P16(cudaMallocAsync((void **)&rows, sizeof(int) * N, st)); frees.add(rows);
    PB_P16(cudaMallocAsync((void **)&cols, sizeof(int) * N, st)); frees.add(cols);
    PB_P16(cudaMallocAsync((void **)&idx, sizeof(int) * N, st)); frees.add(idx);
    PB_P16(cudaMallocAsync((void **)&order, sizeof(int) * N, st)); frees.add(order);
    PB_P16(cudaMallocAsync((void **)&counts, sizeof(int) * 4, st)); frees.add(counts);
    PB_P16(cudaMallocAsync((void **)&keys, sizeof(unsigned long long) * N, st)); frees.add(keys);
    PB_P16(cudaMallocAsync((void **)&keys_sorted, sizeof(unsigned long long) * N, st)); frees.add(keys_sorted);
    PB_P16(cudaMemsetAsync(counts, 0, sizeof(int) * 4, st));
    P16Setup q;
    memset(&q, 0, sizeof q);
    q.alg = m->alg; q.open = m->open; q.gap = m->gap; q.mmax = mmax; q.mmin = mmin; q.nitems = N;
    q.nt = dbmode ? b->npairs : 0;
    q.max_cols = 65535;
    q.qlen = dbmode ? nullptr : b->d_qlen;
    q.prof_qlen = d_pql;
    q.tlen = b->d_tlen;
    q.qlim = b->d_qlim; q.tlim = b->d_tlim;
    q.group = dbmode ? nullptr : group;
    q.intra_mask = intra_mask;
    k_p16_setup<<<(N + 255) / 256, 256, 0, st>>>(q, rows, cols, keys, idx, counts);
    pb_diag_count_launch(1);
    size_t sort_bytes = 0;
    void *sort_tmp = nullptr;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, sort_bytes, keys, keys_sorted, idx, order, N, 0, 64, st);
    PB_P16(cudaMallocAsync(&sort_tmp, sort_bytes, st));
    frees.add(sort_tmp);
    cub::DeviceRadixSort::SortPairsDescending(sort_tmp, sort_bytes, keys, keys_sorted, idx, order, N, 0, 64, st);
    int nelig = 0;
    PB_P16(cudaMemcpyAsync(&nelig, counts, sizeof(int), cudaMemcpyDeviceToHost, st));
    PB_P16(cudaStreamSynchronize(st));
    /* the ineligible items (sorted last) start the rest list */
    if (N - nelig > 0) {
        k_copy_int<<<(N - nelig + 255) / 256, 256, 0, st>>>(order + nelig, N - nelig, d_rest);
        pb_diag_count_launch(1);
    }
    int nrest = N - nelig;
    /* grouped batches: every group starts a task */
    int nslots = nelig;
    int *porder = order;
    if (nelig > 0 && (dbmode || group)) {
        int *head = nullptr, *gid = nullptr, *gstart = nullptr, *pcount = nullptr, *pstart = nullptr, *iota = nullptr;
        int ng = 0, last_start = 0, last_count = 0;
        PB_P16(cudaMallocAsync((void **)&head, sizeof(int) * nelig, st)); frees.add(head);
        PB_P16(cudaMallocAsync((void **)&gid, sizeof(int) * nelig, st)); frees.add(gid);
        PB_P16(cudaMallocAsync((void **)&gstart, sizeof(int) * nelig, st)); frees.add(gstart);
        PB_P16(cudaMallocAsync((void **)&pcount, sizeof(int) * nelig, st)); frees.add(pcount);
        PB_P16(cudaMallocAsync((void **)&pstart, sizeof(int) * nelig, st)); frees.add(pstart);
        PB_P16(cudaMallocAsync((void **)&iota, sizeof(int) * nelig, st)); frees.add(iota);
        k_pad_heads<<<(nelig + 255) / 256, 256, 0, st>>>(keys_sorted, nelig, head);
        k_iota_int<<<(nelig + 255) / 256, 256, 0, st>>>(iota, nelig);
        pb_diag_count_launch(2);
        size_t b1 = 0, b2 = 0, b3 = 0;
        void *tmp = nullptr;
        PB_P16(cub::DeviceScan::InclusiveSum(nullptr, b1, head, gid, nelig, st));
        PB_P16(cub::DeviceSelect::Flagged(nullptr, b2, iota, head, gstart, counts + 2, nelig, st));
        PB_P16(cub::DeviceScan::ExclusiveSum(nullptr, b3, pcount, pstart, nelig, st));
        const size_t tb = std::max(b1, std::max(b2, b3));
        PB_P16(cudaMallocAsync(&tmp, tb, st)); frees.add(tmp);
        size_t b = tb;
        PB_P16(cub::DeviceScan::InclusiveSum(tmp, b, head, gid, nelig, st));
        b = tb;
        PB_P16(cub::DeviceSelect::Flagged(tmp, b, iota, head, gstart, counts + 2, nelig, st));
        PB_P16(cudaMemcpyAsync(&ng, counts + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
        PB_P16(cudaStreamSynchronize(st));
        k_pad_counts<<<(ng + 255) / 256, 256, 0, st>>>(gstart, ng, nelig, pcount);
        pb_diag_count_launch(1);
        b = tb;
        PB_P16(cub::DeviceScan::ExclusiveSum(tmp, b, pcount, pstart, ng, st));
        PB_P16(cudaMemcpyAsync(&last_start, pstart + ng - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        PB_P16(cudaMemcpyAsync(&last_count, pcount + ng - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        PB_P16(cudaStreamSynchronize(st));
        nslots = last_start + last_count;
        PB_P16(cudaMallocAsync((void **)&porder, sizeof(int) * (size_t)nslots, st)); frees.add(porder);
        PB_P16(cudaMemsetAsync(porder, 0xff, sizeof(int) * (size_t)nslots, st));
        k_pad_scatter<<<(nelig + 255) / 256, 256, 0, st>>>(order, nelig, gid, gstart, pstart, porder);
        pb_diag_count_launch(1);
    }
    if (nelig > 0) {
        const int ntasks = (nslots + 31) / 32;
        P16Params p;
        memset(&p, 0, sizeof p);
        p.alg = m->alg; p.sgflags = m->sgflags; p.open = m->open; p.gap = m->gap; p.mmax = mmax; p.mmin = mmin;
        p.nletters = L; p.nitems = nslots; p.order = porder; p.rows = rows; p.cols = cols;
        p.mat8 = d_mat8;
        p.qall = b->d_qall; p.qoff = b->d_qoff; p.profs = d_profs; p.nt = dbmode ? b->npairs : 0;
        p.targets = b->d_targets; p.toff = b->d_toff;
        p.out = out;
        p.ops = d_ops; p.ops_off = d_ops_off; p.path_info = d_path_info;
        int *twmax = nullptr, *tnpass = nullptr, *tshared = nullptr;
        long long *tckpt = nullptr;
        PB_P16(cudaMallocAsync((void **)&twmax, sizeof(int) * ntasks, st)); frees.add(twmax);
        PB_P16(cudaMallocAsync((void **)&tnpass, sizeof(int) * ntasks, st)); frees.add(tnpass);
        PB_P16(cudaMallocAsync((void **)&tshared, sizeof(int) * ntasks, st)); frees.add(tshared);
        PB_P16(cudaMallocAsync((void **)&tckpt, sizeof(long long) * ntasks, st)); frees.add(tckpt);
        k_p16_tasks<<<(ntasks * 32 + 255) / 256, 256, 0, st>>>(p, ntasks, dbmode ? nullptr : group, twmax, tnpass,
                                                               tshared, tckpt, ckpt ? 1 : 0);
        pb_diag_count_launch(1);
        std::vector<int> hw(ntasks), hn(ntasks), hs(ntasks);
        std::vector<long long> hb(ntasks);
        PB_P16(cudaMemcpyAsync(hw.data(), twmax, sizeof(int) * ntasks, cudaMemcpyDeviceToHost, st));
        PB_P16(cudaMemcpyAsync(hn.data(), tnpass, sizeof(int) * ntasks, cudaMemcpyDeviceToHost, st));
        PB_P16(cudaMemcpyAsync(hs.data(), tshared, sizeof(int) * ntasks, cudaMemcpyDeviceToHost, st));
        PB_P16(cudaMemcpyAsync(hb.data(), tckpt, sizeof(long long) * ntasks, cudaMemcpyDeviceToHost, st));
        PB_P16(cudaStreamSynchronize(st));
        int maxlen = 0;
        for (int t = 0; t < ntasks; ++t) maxlen = hw[t] > maxlen ? hw[t] : maxlen;
        /* task order: most work first */
        std::vector<int> torder(ntasks);
        for (int t = 0; t < ntasks; ++t) torder[t] = t;
        std::stable_sort(torder.begin(), torder.end(), [&](int x, int y) {
            return (long long)hn[x] * (hw[x] + 1) > (long long)hn[y] * (hw[y] + 1);
        });
        size_t all_u4 = 0;
        for (int t = 0; t < ntasks; ++t) all_u4 += (size_t)hb[t];
        /* Chunks of like make-up: chunk c takes tasks c, c + nch, ... of the
         * order, so that each ends on small tasks (524 k protein pairs in two
         * chunks: 84.2 ms when the first took the largest tasks, 80.7 so). */
        const int nch = ckpt ? (int)p16_chunks((size_t)ntasks, all_u4 * sizeof(uint4)) : 1;
        std::vector<int> cut(nch + 1, 0);
        if (nch > 1) {
            std::vector<int> dealt;
            dealt.reserve(ntasks);
            for (int c = 0; c < nch; ++c) {
                for (int t = c; t < ntasks; t += nch) dealt.push_back(torder[t]);
                cut[c + 1] = (int)dealt.size();
            }
            torder.swap(dealt);
        }
        cut[nch] = ntasks;
        /* what a chunk may take; halved when its allocation fails */
        size_t budget_u4 = all_u4 / nch + (size_t)*std::max_element(hb.begin(), hb.end()) * 2;
        /* launch shapes and the pass-boundary buffers, sized for the larger grid */
        int dev = 0, nsm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        const bool bias = m->open >= m->gap && mmax + m->open <= 127 && mmin + m->open >= -128;
        int grid[2] = {0, 0}, warps[2] = {0, 0};
        size_t smem[2] = {0, 0};
        p16_kernel_t kern[2];
        for (int sh = 0; sh < 2; ++sh) {
            warps[sh] = p16_warps(sh == 1, L);
            smem[sh] = p16_smem(sh == 1, L, d_mat8 != nullptr);
            kern[sh] = bias ? pick<true>(m->alg, ckpt, ends_on, sh == 1, warps[sh])
                            : pick<false>(m->alg, ckpt, ends_on, sh == 1, warps[sh]);
            int per_sm = 0;
            pb_raise_smem((const void *)kern[sh], (int)smem[sh]);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern[sh], warps[sh] * 32, smem[sh]);
            grid[sh] = (per_sm < 1 ? 1 : per_sm) * nsm;
        }
        const size_t rwarps = (size_t)std::max(grid[0] * warps[0], grid[1] * warps[1]);
        uint32_t *scratch = nullptr;
        PB_P16(cudaMallocAsync((void **)&scratch, ckpt ? 256 : sizeof(uint32_t) * (size_t)(maxlen + 8) * 32 * rwarps, st));
        frees.add(scratch);
        p.scratch = scratch;
        p.colsave = nullptr;
        if (ends_on && m->alg == PB_SW) {
            PB_P16(cudaMallocAsync((void **)&p.colsave, sizeof(uint4) * (P16_R / 2) * 32 * rwarps, st));
            frees.add(p.colsave);
        }
        p.maxlen = maxlen;
        p.task_wmax = twmax; p.task_npass = tnpass; p.task_ckpt = tckpt; p.out2 = out2;
        int *d_tlist = nullptr, *d_counter = nullptr;
        PB_P16(cudaMallocAsync((void **)&d_tlist, sizeof(int) * ntasks, st)); frees.add(d_tlist);
        PB_P16(cudaMallocAsync((void **)&d_counter, sizeof(int) * 2, st)); frees.add(d_counter);
        uint4 *ckbuf = nullptr;
        size_t ck_cap = 0;
        std::vector<long long> hoff(ntasks, 0);
        int t0 = 0;
        while (t0 < ntasks) {
            /* the chunk [t0, t1) of torder, its tasks listed shared-first */
            int t1 = t0;
            size_t used = 0;
            const int t_end = *std::upper_bound(cut.begin(), cut.end(), t0);
            while (t1 < t_end && (t1 == t0 || used + (size_t)hb[torder[t1]] <= budget_u4)) used += (size_t)hb[torder[t1++]];
            std::vector<int> lst[2];
            for (int k = t0; k < t1; ++k) lst[hs[torder[k]] ? 1 : 0].push_back(torder[k]);
            size_t off = 0;
            for (int k = t0; k < t1; ++k) { hoff[torder[k]] = (long long)off; off += (size_t)hb[torder[k]]; }
            if (ckpt && off > ck_cap) {
                if (ckbuf) cudaFreeAsync(ckbuf, st);
                ckbuf = nullptr;
                ck_cap = 0;
                if (cudaMallocAsync((void **)&ckbuf, sizeof(uint4) * (off + 1), st) != cudaSuccess) {
                    ckbuf = nullptr;
                    cudaGetLastError();
                    if (t1 - t0 > 1) { budget_u4 = off / 2; continue; }
                    fprintf(stderr, "pb_pair16: checkpoints of %zu bytes failed\n", sizeof(uint4) * (off + 1));
                    return -1;
                }
                ck_cap = off;
            }
            p.ckpt = ckbuf;
            PB_P16(cudaMemcpyAsync(tckpt, hoff.data(), sizeof(long long) * ntasks, cudaMemcpyHostToDevice, st));
            const int n1 = (int)lst[1].size(), n0 = (int)lst[0].size();
            std::vector<int> all(lst[1]);
            all.insert(all.end(), lst[0].begin(), lst[0].end());
            PB_P16(cudaMemcpyAsync(d_tlist, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice, st));
            for (int sh = 1; sh >= 0; --sh) {
                const int nl = sh ? n1 : n0;
                if (!nl) continue;
                const int *tl = d_tlist + (sh ? 0 : n1);
                int g = grid[sh];
                const int need = (nl + warps[sh] - 1) / warps[sh];
                if (g > need) g = need;
                PB_P16(cudaMemsetAsync(d_counter, 0, sizeof(int), st));
                kern[sh]<<<g, warps[sh] * 32, smem[sh], st>>>(p, tl, nl, d_counter);
                pb_diag_count_launch(1);
                PB_P16(cudaGetLastError());
            }
            if (ckpt) {
                const int mode = paths ? 2 : out2 ? 1 : 0;
                const p16_trace_t tk = bias ? pick_trace<true>(m->alg, mode) : pick_trace<false>(m->alg, mode);
                const size_t tsm = (d_mat8 ? (((size_t)L * L + 15) & ~(size_t)15) : 0) +
                                   (size_t)P16_TR_WARPS * (p16_ck(m->alg) * 512 + (size_t)L * 1024);
                int per_sm = 0;
                pb_raise_smem((const void *)tk, (int)tsm);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tk, P16_TR_WARPS * 32, tsm);
                const int nl = (int)all.size();
                const int g = std::min((per_sm < 1 ? 1 : per_sm) * nsm, (nl + P16_TR_WARPS - 1) / P16_TR_WARPS);
                PB_P16(cudaMemsetAsync(d_counter, 0, sizeof(int), st));
                tk<<<g, P16_TR_WARPS * 32, tsm, st>>>(job, p, d_tlist, nl, prefix ? ends : out, d_counter);
                pb_diag_count_launch(1);
                PB_P16(cudaGetLastError());
            }
            /* the host vectors handed to the copies above change next chunk */
            PB_P16(cudaStreamSynchronize(st));
            t0 = t1;
        }
        if (ckbuf) cudaFreeAsync(ckbuf, st);
        /* items whose width verdicts need exact extremes */
        if (!prefix) {
            PB_P16(cudaMemsetAsync(counts + 1, 0, sizeof(int), st));
            k_p16_check<<<(nslots + 255) / 256, 256, 0, st>>>(job, p, d_rest + nrest, counts + 1);
            pb_diag_count_launch(1);
            int nx = 0;
            PB_P16(cudaMemcpyAsync(&nx, counts + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
            PB_P16(cudaStreamSynchronize(st));
            nrest += nx;
        }
    }
    *n_rest = nrest;
    PB_P16(cudaStreamSynchronize(st));
    return 0;
}

/* --- the intra-task wavefront kernel on a subset (global score-only) -------- */

namespace {

__global__ void k_wave_fill(pb_job job, const int *__restrict__ list, int n, const int *__restrict__ score,
                            const int *__restrict__ qlen, const int *__restrict__ tlen, pb_pair_out *__restrict__ out,
                            int *__restrict__ rest, int *__restrict__ nrest)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int item = list[k];
    const int rows = qlen[k], cols = tlen[k];
    const P16Bounds bd = p16_bounds(PB_NW, rows, cols, job.mode.open, job.mode.gap, job.mode.mmax, job.mode.mmin);
    pb_pair_out o;
    o.score = score[k]; o.end_query = rows - 1; o.end_ref = cols - 1;
    o.matches = o.similar = o.length = 0;
    o.max_h = bd.ub;
    o.min_h_real = bd.lb; o.min_f_real = bd.lb - job.mode.open; o.max_stat_real = ((rows + 31) & ~31) + cols;
    for (int x = 0; x < 3; ++x) { o.min_h_pad[x] = bd.lb; o.max_stat_pad[x] = o.max_stat_real; o.min_f_pad[x] = bd.lb - job.mode.open; }
    o.status = PB_ST_BOUNDED;
    out[item] = o;
    if (!p16_definite(job, o, rows, cols)) rest[atomicAdd(nrest, 1)] = item;
}

__global__ void k_gather_pairs(const int *__restrict__ list, int n, const int64_t *__restrict__ qoff,
                               const int *__restrict__ qlen, const int64_t *__restrict__ toff,
                               const int *__restrict__ tlen, int64_t *__restrict__ gqoff, int *__restrict__ gqlen,
                               int64_t *__restrict__ gtoff, int *__restrict__ gtlen)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int item = list[k];
    gqoff[k] = qoff[item]; gqlen[k] = qlen[item];
    gtoff[k] = toff[item]; gtlen[k] = tlen[item];
}

}  // namespace

bool wave_ok(const pb_job &job, const pb_batch *b)
{
    return job.mode.alg == PB_NW && !job.mode.stats && b->nprofs == 0 && b->d_mat && !b->d_qlim && !b->d_tlim &&
           b->msize <= 32 && b->mmax <= 127 && b->mmin >= -127;
}

int wave_subset(const pb_job &job, const pb_batch *b, const int *d_list, int n, pb_pair_out *out, int *d_rest2,
                int *n_rest2, cudaStream_t st)
{
    *n_rest2 = 0;
    if (n <= 0) return 0;
    P16Frees frees(st);
    int64_t *gq = nullptr, *gt = nullptr;
    int *gql = nullptr, *gtl = nullptr, *sc = nullptr, *cnt = nullptr;
    PB_P16(cudaMallocAsync((void **)&gq, sizeof(int64_t) * n, st)); frees.add(gq);
    PB_P16(cudaMallocAsync((void **)&gt, sizeof(int64_t) * n, st)); frees.add(gt);
    PB_P16(cudaMallocAsync((void **)&gql, sizeof(int) * n, st)); frees.add(gql);
    PB_P16(cudaMallocAsync((void **)&gtl, sizeof(int) * n, st)); frees.add(gtl);
    PB_P16(cudaMallocAsync((void **)&sc, sizeof(int) * n, st)); frees.add(sc);
    PB_P16(cudaMallocAsync((void **)&cnt, sizeof(int), st)); frees.add(cnt);
    k_gather_pairs<<<(n + 255) / 256, 256, 0, st>>>(d_list, n, b->d_qoff, b->d_qlen, b->d_toff, b->d_tlen, gq, gql,
                                                    gt, gtl);
    pb_diag_count_launch(1);
    std::vector<int> hl(n), hm((size_t)b->msize * b->msize);
    PB_P16(cudaMemcpyAsync(hl.data(), gtl, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    PB_P16(cudaMemcpyAsync(hm.data(), b->d_mat, sizeof(int) * hm.size(), cudaMemcpyDeviceToHost, st));
    PB_P16(cudaMemsetAsync(cnt, 0, sizeof(int), st));
    PB_P16(cudaStreamSynchronize(st));
    int maxlen = 0;
    for (int x : hl) maxlen = x > maxlen ? x : maxlen;
    if (pb_cuda_nw_long(n, job.mode.open, job.mode.gap, hm.data(), b->msize, b->d_qall, gq, gql, b->d_targets, gt,
                        gtl, nullptr, nullptr, maxlen, sc) != 0)
        return -1;
    PB_P16(cudaDeviceSynchronize());
    k_wave_fill<<<(n + 255) / 256, 256, 0, st>>>(job, d_list, n, sc, gql, gtl, out, d_rest2, cnt);
    pb_diag_count_launch(1);
    PB_P16(cudaMemcpyAsync(n_rest2, cnt, sizeof(int), cudaMemcpyDeviceToHost, st));
    PB_P16(cudaStreamSynchronize(st));
    return 0;
}

/* --- the exact kernel on a subset of a batch's items ------------------------ */

namespace {

__global__ void k_gather_items(const int *__restrict__ list, int n, int nt, const int64_t *__restrict__ toff,
                               const int *__restrict__ tlen, const int64_t *__restrict__ qoff,
                               const int *__restrict__ qlen, const int *__restrict__ qlim,
                               const int *__restrict__ tlim, int64_t *__restrict__ g_toff, int *__restrict__ g_tlen,
                               int64_t *__restrict__ g_qoff, int *__restrict__ g_qlen, int *__restrict__ g_pidx,
                               int *__restrict__ g_qlim, int *__restrict__ g_tlim)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int item = list[k];
    const int ti = nt ? item % nt : item;
    g_toff[k] = toff[ti];
    g_tlen[k] = tlen[ti];
    if (nt) g_pidx[k] = item / nt;
    else { g_qoff[k] = qoff[item]; g_qlen[k] = qlen[item]; }
    if (qlim) g_qlim[k] = qlim[item];
    if (tlim) g_tlim[k] = tlim[item];
}

__global__ void k_scatter_items(const pb_pair_out *__restrict__ src, const int *__restrict__ list, int n,
                                pb_pair_out *__restrict__ dst)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[list[k]] = src[k];
}

}  // namespace

int exact_subset(const pb_batch *b, const int *d_list, int n, int stats, int pad_rows, pb_pair_out *out,
                 cudaStream_t st)
{
    if (n <= 0) return 0;
    const bool dbmode = b->nprofs > 0;
    P16Frees frees(st);
    int64_t *g_toff = nullptr, *g_qoff = nullptr;
    int *g_tlen = nullptr, *g_qlen = nullptr, *g_pidx = nullptr, *g_qlim = nullptr, *g_tlim = nullptr;
    pb_pair_out *tmp = nullptr;
    PB_P16(cudaMallocAsync((void **)&g_toff, sizeof(int64_t) * n, st)); frees.add(g_toff);
    PB_P16(cudaMallocAsync((void **)&g_tlen, sizeof(int) * n, st)); frees.add(g_tlen);
    PB_P16(cudaMallocAsync((void **)&tmp, sizeof(pb_pair_out) * n, st)); frees.add(tmp);
    if (dbmode) {
        PB_P16(cudaMallocAsync((void **)&g_pidx, sizeof(int) * n, st)); frees.add(g_pidx);
    } else {
        PB_P16(cudaMallocAsync((void **)&g_qoff, sizeof(int64_t) * n, st)); frees.add(g_qoff);
        PB_P16(cudaMallocAsync((void **)&g_qlen, sizeof(int) * n, st)); frees.add(g_qlen);
    }
    if (b->d_qlim) { PB_P16(cudaMallocAsync((void **)&g_qlim, sizeof(int) * n, st)); frees.add(g_qlim); }
    if (b->d_tlim) { PB_P16(cudaMallocAsync((void **)&g_tlim, sizeof(int) * n, st)); frees.add(g_tlim); }
    k_gather_items<<<(n + 255) / 256, 256, 0, st>>>(d_list, n, dbmode ? b->npairs : 0, b->d_toff, b->d_tlen,
                                                    b->d_qoff, b->d_qlen, b->d_qlim, b->d_tlim, g_toff, g_tlen,
                                                    g_qoff, g_qlen, g_pidx, g_qlim, g_tlim);
    pb_diag_count_launch(1);
    PB_P16(cudaStreamSynchronize(st));
    pb_batch s = *b;
    s.npairs = n;
    s.stats = stats;
    s.pad_rows = pad_rows;
    s.d_toff = g_toff; s.d_tlen = g_tlen;
    s.d_qlim = g_qlim; s.d_tlim = g_tlim;
    s.d_out = tmp;
    if (dbmode) s.d_prof_index = g_pidx;
    else { s.d_qoff = g_qoff; s.d_qlen = g_qlen; }
    if (pb_cuda_align_exact(&s) != 0) return -1;
    k_scatter_items<<<(n + 255) / 256, 256, 0, st>>>(tmp, d_list, n, out);
    pb_diag_count_launch(1);
    PB_P16(cudaStreamSynchronize(st));
    return 0;
}

}  // namespace pb

namespace {

/* characters of raw to codes at the same offsets */
__global__ void k_p16_map_into(const uint8_t *__restrict__ raw, uint8_t *__restrict__ codes, int64_t n,
                               const uint8_t *__restrict__ map)
{
    __shared__ uint8_t smap[256];
    for (int k = threadIdx.x; k < 256; k += blockDim.x) smap[k] = map[k];
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        codes[i] = smap[raw[i]];
}

/* What the CIGARs of a slice of a batch are built from and into. */
struct CigarParams {
    int n, sg;
    const uint8_t *ops;             /* steps, at the end of each pair's rows + columns bytes */
    const int64_t *ooff;
    const int *info, *ends;         /* 3 per pair: steps, stop row and column; score and ends */
    const uint8_t *q, *t;           /* characters */
    const int64_t *qoff, *toff;
    const int *qlen, *tlen;
    const uint8_t *upper;           /* toupper of every character */
    uint32_t *cig;                  /* elements, at ooff[k] - cig0 */
    int64_t cig0;
    int *len, *cnt, *beg;           /* elements (-1: no CIGAR), elements to copy, first positions */
};

/*
 * The CIGARs that parasail_result_get_cigar builds (src/cigar_template.c)
 * from the paths, a thread per pair: gaps to the matrix edge where the walk
 * reached it, the steps ('=' or 'X' by the upper-cased characters), a
 * semi-global alignment's end gaps, runs merged. Latency bound on a few
 * hundred dependent steps a thread (40,000 reads of 200: 190 us), where the
 * host took 46 of the call's 53 ms to build results and CIGARs one by one;
 * the call now takes 6.2 ms.
 */
__global__ void k_p16_cigar(CigarParams p)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p.n) return;
    const int steps = p.info[3 * k];
    p.cnt[k] = 0;
    p.len[k] = -1;
    p.beg[2 * k] = p.beg[2 * k + 1] = 0;
    if (steps < 0) return;
    const int lena = p.qlen[k], lenb = p.tlen[k];
    const int end_q = p.ends[3 * k + 1], end_r = p.ends[3 * k + 2];
    const uint8_t *ops = p.ops + p.ooff[k] + lena + lenb - steps;
    const uint8_t *a = p.q + p.qoff[k], *b = p.t + p.toff[k];
    uint32_t *out = p.cig + (p.ooff[k] - p.cig0);
    int i = p.info[3 * k + 1], j = p.info[3 * k + 2], n = 0;
    uint32_t op = 0, run = 0;
    auto add = [&](uint32_t o, int c) {
        if (c <= 0) return;
        if (run && o != op) { out[n++] = (run << 4) | op; run = 0; }
        op = o;
        run += (uint32_t)c;
    };
    /* BAM operations: I 1, D 2, = 7, X 8 */
    int bq = i + 1, br = j + 1;
    if (i < 0 && j >= 0) { add(2u, j + 1); br = 0; }
    else if (j < 0 && i >= 0) { add(1u, i + 1); bq = 0; }
    i += 1;
    j += 1;
    for (int x = 0; x < steps; ++x) {
        const uint8_t o = ops[x];
        if (o == 0) {
            if (i >= lena || j >= lenb) break;
            add(p.upper[a[i]] == p.upper[b[j]] ? 7u : 8u, 1);
            ++i;
            ++j;
        } else if (o == 1) {
            add(1u, 1);
            ++i;
        } else {
            add(2u, 1);
            ++j;
        }
    }
    if (p.sg) {
        if (end_q + 1 == lena) add(2u, lenb - 1 - end_r);
        else if (end_r + 1 == lenb) add(1u, lena - 1 - end_q);
        else return;
    }
    if (run) out[n++] = (run << 4) | op;
    p.len[k] = n;
    p.cnt[k] = n;
    p.beg[2 * k] = bq;
    p.beg[2 * k + 1] = br;
}

/* the pairs' elements side by side, a warp per pair */
__global__ void k_p16_cigar_pack(CigarParams p, const int64_t *__restrict__ coff, uint32_t *__restrict__ out)
{
    const int k = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (k >= p.n) return;
    const uint32_t *cig = p.cig + (p.ooff[k] - p.cig0);
    const int c = p.cnt[k];
    for (int x = lane; x < c; x += 32) out[coff[k] + x] = cig[x];
}

__global__ void k_p16_ends(const pb_pair_out *__restrict__ o, int n, int *__restrict__ se)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    se[3 * k] = o[k].score;
    se[3 * k + 1] = o[k].end_query;
    se[3 * k + 2] = o[k].end_ref;
}

}  // namespace

/* where trace_host puts CIGARs (pb_cuda_trace_cigars_host) */
struct TraceCigars {
    const uint8_t *upper;
    int *len, *beg;
    uint32_t **elems;
};

/* The CIGARs of all pairs, slice by slice: built on the device, packed there,
 * and copied behind those of the slices before. cp holds the batch's device
 * arrays. */
static int trace_cigars(CigarParams cp, int n, const int *h_qlen, const int *h_tlen, const int64_t *h_ooff,
                        const TraceCigars &cig, cudaStream_t st)
{
    pb::P16Frees frees(st);
    size_t most = 0, have = 0;             /* elements: of a slice, on the host so far */
    int widest = 0;                        /* pairs of a slice */
    for (int k0 = 0, k1; k0 < n; k0 = k1) {
        k1 = cigar_slice_end(h_ooff, h_qlen, h_tlen, n, k0, CIGAR_SLICE);
        most = std::max(most, (size_t)(h_ooff[k1 - 1] + h_qlen[k1 - 1] + h_tlen[k1 - 1] - h_ooff[k0]));
        widest = std::max(widest, k1 - k0);
    }
    uint32_t *d_cig = nullptr;
    int *d_len = nullptr;
    int64_t *d_coff = nullptr;
    void *d_tmp = nullptr;
    size_t tmp_bytes = 0;
    /* the sums run in 64 bits, whatever the type of the counts */
    auto scan = [&](int items) {
        return cub::DeviceScan::ExclusiveScan(d_tmp, tmp_bytes, d_len, d_coff, cuda::std::plus<int64_t>{}, (int64_t)0, items, st);
    };
    if (scan(widest + 1) != cudaSuccess) return -1;
    if (cudaMallocAsync((void **)&d_cig, sizeof(uint32_t) * (most + 1), st) == cudaSuccess) frees.add(d_cig);
    if (cudaMallocAsync((void **)&d_len, sizeof(int) * (4 * (size_t)widest + 1), st) == cudaSuccess) frees.add(d_len);
    if (cudaMallocAsync((void **)&d_coff, sizeof(int64_t) * ((size_t)widest + 1), st) == cudaSuccess) frees.add(d_coff);
    if (cudaMallocAsync(&d_tmp, tmp_bytes, st) == cudaSuccess) frees.add(d_tmp);
    if (frees.v.size() != 4) { cudaGetLastError(); return -1; }
    const CigarParams all = cp;
    for (int k0 = 0, k1; k0 < n; k0 = k1) {
        k1 = cigar_slice_end(h_ooff, h_qlen, h_tlen, n, k0, CIGAR_SLICE);
        const int m = k1 - k0;
        /* d_len: [counts, one 0 after them][lengths][first positions] */
        cp.n = m;
        cp.info = all.info + 3 * (size_t)k0; cp.ends = all.ends + 3 * (size_t)k0;
        cp.ooff = all.ooff + k0; cp.qoff = all.qoff + k0; cp.toff = all.toff + k0;
        cp.qlen = all.qlen + k0; cp.tlen = all.tlen + k0;
        cp.cig = d_cig; cp.cig0 = h_ooff[k0];
        cp.cnt = d_len; cp.len = d_len + m + 1; cp.beg = d_len + 2 * (size_t)m + 1;
        int64_t total = 0;
        cudaMemsetAsync(d_len + m, 0, sizeof(int), st);
        k_p16_cigar<<<(m + 63) / 64, 64, 0, st>>>(cp);
        if (scan(m + 1) != cudaSuccess) return -1;
        pb_diag_count_launch(1);
        if (cudaMemcpyAsync(cig.len + k0, cp.len, sizeof(int) * (size_t)m, cudaMemcpyDeviceToHost, st) ||
            cudaMemcpyAsync(cig.beg + 2 * (size_t)k0, cp.beg, sizeof(int) * 2 * (size_t)m, cudaMemcpyDeviceToHost, st) ||
            cudaMemcpyAsync(&total, d_coff + m, sizeof total, cudaMemcpyDeviceToHost, st) ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return -1;
        uint32_t *elems = (uint32_t *)realloc(*cig.elems, sizeof(uint32_t) * (have + (size_t)total + 1));
        if (!elems) return -1;
        *cig.elems = elems;
        uint32_t *d_pack = nullptr;
        if (cudaMallocAsync((void **)&d_pack, sizeof(uint32_t) * (size_t)(total + 1), st) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        const int64_t threads = 32 * (int64_t)m;
        k_p16_cigar_pack<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(cp, d_coff, d_pack);
        pb_diag_count_launch(1);
        cudaError_t e = cudaMemcpyAsync(elems + have, d_pack, sizeof(uint32_t) * (size_t)total, cudaMemcpyDeviceToHost, st);
        cudaFreeAsync(d_pack, st);
        if (e != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) return -1;
        have += (size_t)total;
    }
    return 0;
}

/* Traceback paths of n pairs from host memory (pairs mode: tmpl carries the
 * matrix table on the device): characters copied and mapped on the device,
 * the pair kernels with checkpoints and the traceback, then per pair
 * h_ends[3k..] = score, end_query, end_ref, the steps in
 * h_ops[h_ops_off[k] ..] (written backwards from the end of the pair's
 * qlen + tlen bytes) and h_info[3k..] = steps (-1: the pair is outside the
 * 16-bit bounds of the pair kernels and has no path), stop row, stop
 * column. */
static int trace_host(const pb_job *job, const pb_batch *tmpl, const uint8_t *mapper256,
                      const char *h_q, const int64_t *h_qoff, const int *h_qlen,
                      const char *h_t, const int64_t *h_toff, const int *h_tlen, int n,
                      int *h_ends, uint8_t *h_ops, const int64_t *h_ops_off, int *h_info, const TraceCigars *cig)
{
    if (pb_cuda_init() != 0) return -1;
    if (n <= 0) return 0;
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return -1;
    int rc = 0;
    {
        pb::P16Frees frees(st);
        int64_t qb = 0, tb = 0, ob = 0;
        for (int i = 0; i < n; ++i) {
            qb = std::max(qb, h_qoff[i] + h_qlen[i]);
            tb = std::max(tb, h_toff[i] + h_tlen[i]);
            ob = std::max(ob, h_ops_off[i] + h_qlen[i] + h_tlen[i]);
        }
        uint8_t *d_q = nullptr, *d_t = nullptr, *d_map = nullptr, *d_ops = nullptr;
        uint8_t *d_qraw = nullptr, *d_traw = nullptr;
        int64_t *d_qoff = nullptr, *d_toff = nullptr, *d_ooff = nullptr;
        int *d_qlen = nullptr, *d_tlen = nullptr, *d_info = nullptr, *d_rest = nullptr, *d_se = nullptr;
        pb_pair_out *d_o = nullptr;
        if (cudaMallocAsync((void **)&d_q, qb + 16, st) || cudaMallocAsync((void **)&d_t, tb + 16, st) ||
            cudaMallocAsync((void **)&d_map, 512, st) || cudaMallocAsync((void **)&d_qraw, qb + 16, st) ||
            cudaMallocAsync((void **)&d_traw, tb + 16, st) || cudaMallocAsync((void **)&d_ops, ob + 16, st) ||
            cudaMallocAsync((void **)&d_qoff, sizeof(int64_t) * n, st) ||
            cudaMallocAsync((void **)&d_toff, sizeof(int64_t) * n, st) ||
            cudaMallocAsync((void **)&d_ooff, sizeof(int64_t) * n, st) ||
            cudaMallocAsync((void **)&d_qlen, sizeof(int) * n, st) || cudaMallocAsync((void **)&d_tlen, sizeof(int) * n, st) ||
            cudaMallocAsync((void **)&d_info, sizeof(int) * 3 * (size_t)n, st) ||
            cudaMallocAsync((void **)&d_se, sizeof(int) * 3 * (size_t)n, st) ||
            cudaMallocAsync((void **)&d_rest, sizeof(int) * n, st) ||
            cudaMallocAsync((void **)&d_o, sizeof(pb_pair_out) * n, st))
            rc = -1;
        void *ptrs[] = {d_q, d_t, d_qraw, d_traw, d_map, d_ops, d_qoff, d_toff, d_ooff, d_qlen, d_tlen, d_info, d_se, d_rest, d_o};
        for (void *x : ptrs) frees.add(x);
        if (rc == 0) {
            cudaMemcpyAsync(d_qraw, h_q, qb, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_traw, h_t, tb, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_map, mapper256, 256, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_qoff, h_qoff, sizeof(int64_t) * n, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_toff, h_toff, sizeof(int64_t) * n, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_ooff, h_ops_off, sizeof(int64_t) * n, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_qlen, h_qlen, sizeof(int) * n, cudaMemcpyHostToDevice, st);
            cudaMemcpyAsync(d_tlen, h_tlen, sizeof(int) * n, cudaMemcpyHostToDevice, st);
            cudaMemsetAsync(d_info, 0xff, sizeof(int) * 3 * (size_t)n, st);
            cudaMemsetAsync(d_o, 0, sizeof(pb_pair_out) * n, st);
            if (cig) cudaMemcpyAsync(d_map + 256, cig->upper, 256, cudaMemcpyHostToDevice, st);
            k_p16_map_into<<<296, 256, 0, st>>>(d_qraw, d_q, qb, d_map);
            k_p16_map_into<<<296, 256, 0, st>>>(d_traw, d_t, tb, d_map);
            pb_diag_count_launch(2);
            if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
        }
        if (rc == 0) {
            pb_batch b = *tmpl;
            b.nprofs = 0;
            b.npairs = n;
            b.stats = 0;
            b.d_qall = d_q; b.d_qoff = d_qoff; b.d_qlen = d_qlen;
            b.d_targets = d_t; b.d_toff = d_toff; b.d_tlen = d_tlen;
            b.d_qlim = nullptr; b.d_tlim = nullptr;
            b.d_out = d_o;
            int nrest = 0;
            rc = pb::p16_pass(*job, &b, 0, nullptr, d_o, nullptr, d_rest, &nrest, st, d_ops, d_ooff, d_info);
        }
        if (rc == 0) {
            k_p16_ends<<<(n + 255) / 256, 256, 0, st>>>(d_o, n, d_se);
            pb_diag_count_launch(1);
            if (cudaMemcpyAsync(h_ends, d_se, sizeof(int) * 3 * (size_t)n, cudaMemcpyDeviceToHost, st) ||
                cudaMemcpyAsync(h_info, d_info, sizeof(int) * 3 * (size_t)n, cudaMemcpyDeviceToHost, st) ||
                (!cig && cudaMemcpyAsync(h_ops, d_ops, ob, cudaMemcpyDeviceToHost, st)))
                rc = -1;
        }
        if (rc == 0 && cig) {
            CigarParams cp;
            cp.sg = job->mode.alg == PB_SG;
            cp.ops = d_ops; cp.ooff = d_ooff; cp.info = d_info; cp.ends = d_se;
            cp.q = d_qraw; cp.t = d_traw; cp.qoff = d_qoff; cp.toff = d_toff; cp.qlen = d_qlen; cp.tlen = d_tlen;
            cp.upper = d_map + 256;
            /* (with no path among the pairs there is nothing to build) */
            if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
            int first = 0;
            while (rc == 0 && first < n && h_info[3 * (size_t)first] < 0) ++first;
            if (rc == 0 && first < n) {
                rc = trace_cigars(cp, n, h_qlen, h_tlen, h_ops_off, *cig, st);
            } else if (rc == 0) {
                std::fill(cig->len, cig->len + n, -1);
                std::fill(cig->beg, cig->beg + 2 * (size_t)n, 0);
            }
        }
        if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
    }
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return rc;
}

extern "C" int pb_cuda_trace_pairs_host(const pb_job *job, const pb_batch *tmpl, const uint8_t *mapper256,
                                        const char *h_q, const int64_t *h_qoff, const int *h_qlen,
                                        const char *h_t, const int64_t *h_toff, const int *h_tlen, int n,
                                        int *h_ends, uint8_t *h_ops, const int64_t *h_ops_off, int *h_info)
{
    return trace_host(job, tmpl, mapper256, h_q, h_qoff, h_qlen, h_t, h_toff, h_tlen, n, h_ends, h_ops, h_ops_off,
                      h_info, nullptr);
}

/* The same with the CIGARs instead of the paths: h_len[k] elements of pair k
 * (-1: none), its first positions in h_beg[2k..], the elements of all pairs
 * side by side in *h_elems (malloc'd, the caller's; null when there are none,
 * as it has to be at the call). upper256: toupper of every character.
 * h_ops_off: ascending, pair k's rows + columns after it. */
extern "C" int pb_cuda_trace_cigars_host(const pb_job *job, const pb_batch *tmpl, const uint8_t *mapper256,
                                         const uint8_t *upper256, const char *h_q, const int64_t *h_qoff,
                                         const int *h_qlen, const char *h_t, const int64_t *h_toff, const int *h_tlen,
                                         int n, int *h_ends, const int64_t *h_ops_off, int *h_info, int *h_len,
                                         int *h_beg, uint32_t **h_elems)
{
    const TraceCigars c = {upper256, h_len, h_beg, h_elems};
    return trace_host(job, tmpl, mapper256, h_q, h_qoff, h_qlen, h_t, h_toff, h_tlen, n, h_ends, nullptr, h_ops_off,
                      h_info, &c);
}

/* ---- the schedule table -------------------------------------------------------
 * Which length buckets of global score-only pairs run on the intra-task
 * wavefront kernel (one team of warps per pair) rather than the inter-task
 * pair kernel (one thread per pair). Written by the tuner
 * (parasail_b200/tune.py) as lines "mode bucket max_len inter_gcups
 * intra_gcups winner"; read from $PARASAIL_B200_SCHEDULE, else from
 * schedule.txt beside the library, on first use. */

namespace {

std::once_flag g_sched_once;
std::mutex g_sched_mu;
unsigned g_sched_nw = 0;

int sched_load_file(const char *path, unsigned *mask)
{
    FILE *f = fopen(path, "r");
    if (!f) return -1;
    char line[256], mode[32], win[32];
    unsigned m = 0;
    int bucket, maxlen;
    double a, b;
    while (fgets(line, sizeof line, f)) {
        if (line[0] == '#') continue;
        if (sscanf(line, "%31s %d %d %lf %lf %31s", mode, &bucket, &maxlen, &a, &b, win) == 6 &&
            !strcmp(mode, "nw") && bucket >= 0 && bucket < 32 && !strcmp(win, "intra"))
            m |= 1u << bucket;
    }
    fclose(f);
    *mask = m;
    return 0;
}

void sched_init()
{
    unsigned m = 0;
    const char *env = getenv("PARASAIL_B200_SCHEDULE");
    if (env && *env) {
        if (sched_load_file(env, &m) == 0) g_sched_nw = m;
        return;
    }
    Dl_info info;
    if (dladdr((void *)&sched_init, &info) && info.dli_fname) {
        std::string dir(info.dli_fname);
        const size_t slash = dir.rfind('/');
        dir = slash == std::string::npos ? std::string(".") : dir.substr(0, slash);
        if (sched_load_file((dir + "/schedule.txt").c_str(), &m) == 0) g_sched_nw = m;
    }
}

}  // namespace

namespace pb {

unsigned pb_schedule_nw_mask()
{
    std::call_once(g_sched_once, sched_init);
    std::lock_guard<std::mutex> lk(g_sched_mu);
    return g_sched_nw;
}

}  // namespace pb

extern "C" unsigned parasail_b200_schedule_get(void)
{
    return pb::pb_schedule_nw_mask();
}

extern "C" void parasail_b200_schedule_set(unsigned intra_mask)
{
    std::call_once(g_sched_once, sched_init);
    std::lock_guard<std::mutex> lk(g_sched_mu);
    g_sched_nw = intra_mask;
}
