/*
 * pb_sw16.cu -- Smith-Waterman score-only kernel in packed int16x2 lanes.
 *
 * Inter-task schedule: every thread aligns one query/target pair; a warp
 * takes 32 targets of similar length (targets are sorted by length) against
 * one query, and a persistent grid pulls such tasks for all queries of the
 * batch, longest first. The query is processed in passes of 2 x 16 rows:
 * the low 16-bit half of every register holds strip A (rows r0..r0+15) at
 * target column j, the high half strip B (rows r0+16..r0+31) at column j-1,
 * so strip B reads strip A's bottom row from the previous iteration and both
 * halves of one DPX instruction always do useful, independent work. A pass
 * hands its bottom row (H and the vertical-gap value F, 16 bits each) to the
 * next pass through a per-warp buffer laid out [column][lane]: one
 * contiguous 128-byte transaction per warp access. Each warp stages the
 * int8 scores of its pass's 32 rows in shared memory; a column's 16 + 16
 * scores are two 16-byte loads expanded to int16x2 words by sign-extending
 * byte permutes. The recurrence is written so that two DPX operations per
 * row sit on the column's dependency chain (F = viaddmax(H_up, -open,
 * F_up - gap) and H = max(A, F), with A = max(H_diag + s, E, 0) computed off
 * the chain), and one in the biased form (k_sw16<true>, open >= gap): the
 * registers hold H - open and the profile s + open, and
 * F(i+1) = max(F(i) - gap, A(i) - open) since F(i) - open <= F(i) - gap.
 *
 * Semantics: the Smith-Waterman recurrence of the reference's striped/scan
 * kernels and of src/sw.c:131-158, with its end-position rule (first column
 * reaching the maximum, then the smallest query row; src/sw.c:150-158,
 * src/sw_striped_avx2_256_16.c:350-409). The 16-bit lanes hold exact values
 * while every H stays below 32767 - max(matrix) - 1; a pair that reaches
 * that bound is reported with PB_ST_OVERFLOW16 and must be rerun by the
 * exact 32-bit kernel. E and F start at -open, which is equivalent to -inf in
 * Smith-Waterman (H is clamped at 0) and keeps E - gap, F - gap in range.
 */
#include <cstdio>
#include <cstdint>
#include <climits>
#include <cuda_runtime.h>

#include "pb_codes.h"
#include "pb_cuda.h"
#include "pb_kernels.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <vector>
#include <mutex>

namespace pb {

static constexpr int SW16_R = 16;          /* query rows per strip (two strips per pass) */
static constexpr int SW16_WARPS = 8;       /* warps per block */
static constexpr int WAVE16_WARPS = 4;     /* warps per block of k_sw_wave16 */
static constexpr int SW16_ROW = 48;        /* bytes between two letters' scores in a warp's slice */

/* Packs two signed bytes (byte k of a and of b) into one int16x2 word:
 * low half from a, high half from b, each sign-extended (prmt sign mode). */
template <int K>
__device__ __forceinline__ uint32_t pack_pair(uint32_t a, uint32_t b)
{
    constexpr uint32_t sel = (K) | ((K | 8) << 4) | ((4 + K) << 8) | (((4 + K) | 8) << 12);
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

__device__ __forceinline__ int s16lo(uint32_t x) { return (int)(int16_t)(x & 0xffffu); }
__device__ __forceinline__ int s16hi(uint32_t x) { return (int)(int16_t)(x >> 16); }
__device__ __forceinline__ uint32_t splat16(int v) { return ((uint32_t)(uint16_t)v) | ((uint32_t)(uint16_t)v << 16); }

struct Sw16Best {
    int score, i, j;
};

/* higher score, then smaller column; an equal column keeps the earlier
 * (smaller) row, which was folded first (scores are positive, a best of 0
 * is none) */
__device__ __forceinline__ void fold_best(Sw16Best &best, const Sw16Best &s)
{
    if (s.j >= 0 && (s.score > best.score || (s.score == best.score && s.j < best.j))) best = s;
}

/* Does a sequence hold a code outside an alphabet of L letters? Aligned
 * 16-byte loads, of those blocks only that hold a byte of the sequence. A call
 * of its own: inlined it changed the register allocation of k_sw16's column
 * loop, 5% on the large search. */
__device__ __noinline__ bool outside_alphabet(const uint8_t *seq, int n, int L)
{
    if (n <= 0) return false;
    const uintptr_t p = reinterpret_cast<uintptr_t>(seq);
    const uint4 *b = reinterpret_cast<const uint4 *>(p & ~(uintptr_t)15);
    const int first = (int)(p & 15), end = first + n, last = (end - 1) >> 4;
    uint32_t m = 0u;
    /* word w of the blocks; its bytes before `first` and from `end` on are not
     * the sequence's */
    auto edge = [&](uint32_t x, int w) {
        const int skip = first - 4 * w, keep = end - 4 * w;
        uint32_t o = codes_outside(x, L);
        if (skip > 0) o &= skip >= 4 ? 0u : 0xffffffffu << (8 * skip);
        if (keep < 4) o &= keep <= 0 ? 0u : 0xffffffffu >> (8 * (4 - keep));
        m |= o;
    };
    const uint4 x0 = __ldg(b), x1 = __ldg(b + last);
    edge(x0.x, 0); edge(x0.y, 1); edge(x0.z, 2); edge(x0.w, 3);
    edge(x1.x, 4 * last); edge(x1.y, 4 * last + 1); edge(x1.z, 4 * last + 2); edge(x1.w, 4 * last + 3);
#pragma unroll 8
    for (int k = 1; k < last; ++k) {
        const uint4 x = __ldg(b + k);
        m |= codes_outside(x.x, L) | codes_outside(x.y, L) | codes_outside(x.z, L) | codes_outside(x.w, L);
    }
    return m != 0u;
}

/*
 * What bounds it: the ALU pipe, which takes the DPX operations and byte
 * permutes at half rate (64 lanes per SM and cycle): 5.5 per row of two
 * cells (byte permute, E, A, F, H and half a three-way maximum; the add of
 * -open issues on the FMA pipe beside them). So the column loop carries
 * little else: four columns per iteration without a branch for each (the
 * columns past the longest target, three at most, meet letter 0 and count
 * for nothing), targets read by words, pass boundaries at pointers that
 * advance by constants with the first pass reading none.
 * The pass's 32 rows of scores are staged per warp as [letter][48 bytes]:
 * 16-byte loads at an odd multiple of 16 bytes fall on all eight bank
 * groups (at the profiles' own stride, a multiple of 64, the kernel took
 * 1.07 to 1.17 times as long), and the launch holds any number of queries of
 * any length, where whole profiles in shared memory ended at 200 KB.
 * 5 queries (100-2000) x 200,000 targets (2.7e11 cells): 102.0 -> 54.9 ms,
 * 4,950 GCUPS, ALU pipe 84% busy; 40 queries (median 270) x 10,000 targets:
 * 28 ms in four launches of whole profiles -> 11.9 ms in one.
 */
template <bool BIAS>
__global__ void __launch_bounds__(SW16_WARPS * 32, 2)
k_sw16(Sw16Params p, int *task_counter)
{
    extern __shared__ __align__(16) int8_t s_slices[];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    int8_t *slice = s_slices + (size_t)wid * p.nletters * SW16_ROW;
    /* the block's SW16_WARPS buffers: warp w's is team_buf + w * maxlen * 32;
     * entry c + 1 is strip B's bottom row at column c, H in the low and F in
     * the high 16 bits */
    uint32_t *team_buf = p.scratch + (size_t)blockIdx.x * SW16_WARPS * p.maxlen * 32 + lane;
    const uint32_t gapO = splat16(-p.open);
    const uint32_t gapE = splat16(-p.gap);
    /* BIAS: the H registers, the pass buffer, the column maxima and the
     * best-so-far hold H - open, so "H = 0" reads as -open */
    const uint32_t zeroH = BIAS ? gapO : 0u;
    const int bias = BIAS ? p.open : 0;
    const uint32_t b4 = BIAS ? 0x01010101u * (uint32_t)(uint8_t)p.open : 0u;
    /* team tasks: the tasks at the front of the list (those that one warp
     * alone would finish last) are run by all warps of a block together,
     * pass k of the task on warp k % SW16_WARPS; a pass reads the previous
     * one's bottom row from that warp's buffer, published every 8 columns
     * through s_prog (generation-tagged, so that it only grows). A pass then
     * runs 11 to 18 columns behind its predecessor; at 32 columns the lag of
     * 64 left the eight warps waiting on targets of less than 512 residues. */
    __shared__ volatile long long s_prog[SW16_WARPS];
    __shared__ int s_task;
    __shared__ Sw16Best s_best[SW16_WARPS][32];
    volatile int *verr = task_counter + 2;
    /* this thread's copies of its strips' best columns: A's 16 words, then B's */
    uint4 *save = p.colsave + ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * (SW16_R / 2);
    bool team = p.nteam > 0;

    /* warp tasks: without team tasks the first of each warp block-strided,
     * so that the largest ones (the list is sorted by cost) are spread one
     * per block instead of landing on the first blocks' SMs; then from the
     * shared counter */
    const int nstatic = p.nteam > 0 ? 0 : gridDim.x * SW16_WARPS;
    bool first = nstatic > 0;
    for (;;) {
        int task = 0, trank = 0, tsize = 1;
        if (team) {
            __syncthreads();
            if (threadIdx.x == 0) s_task = atomicAdd(task_counter + 1, 1);
            if (threadIdx.x < SW16_WARPS) s_prog[threadIdx.x] = 0;
            __syncthreads();
            task = s_task;
            if (task >= p.nteam) { team = false; continue; }
            trank = wid;
            tsize = SW16_WARPS;
        } else {
            if (first) {
                task = blockIdx.x + gridDim.x * wid;
                first = false;
            } else {
                if (lane == 0) task = p.nteam + nstatic + atomicAdd(task_counter, 1);
                task = __shfl_sync(0xffffffffu, task, 0);
            }
            if (task >= p.ntasks) break;
        }
        uint32_t *out_buf = team_buf + (size_t)(team ? trank : wid) * p.maxlen * 32;
        const uint32_t *in_buf = team ? team_buf + (size_t)((trank + tsize - 1) % tsize) * p.maxlen * 32 : out_buf;
        const Sw16Task T = p.tasks[task];
        const Sw16Query Q = p.queries[T.q];
        const int s = T.first + lane;
        const bool valid = s < p.npairs;
        const int pid = valid ? p.order[s] : 0;
        int len = valid ? p.tlen[pid] : 0;
        const uint8_t *tseq = p.targets + (valid ? p.toff[pid] : 0);
        /* A code outside the alphabet would index past the slice: such a
         * target counts as empty here and its pair goes to the exact kernel,
         * which reads the code as letter 0. Looked for once per task: 5
         * queries x 200,000 targets 54.6 -> 54.9 ms, 100 rows x 20,000 targets
         * 277 -> 285 us (a check of four codes in the column loop: 55.9 ms
         * without a branch, 57.3 with one). */
        if (outside_alphabet(tseq, len, p.nletters)) len = 0;
        int wmax = len;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wmax = max(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
        const int ql = Q.qlen;

        Sw16Best best = {0, 0, 0};

        const long long stride = (long long)wmax + 1;
        for (int r0 = 2 * SW16_R * trank; r0 < ql; r0 += 2 * SW16_R * tsize) {
            const int sp = r0 / (2 * SW16_R);            /* pass index */
            /* the pass's scores of every letter (BIAS: + open; the host
             * checked that it stays in int8) */
            __syncwarp();
            for (int x = lane; x < 2 * p.nletters; x += 32) {
                int4 v = __ldg(reinterpret_cast<const int4 *>(Q.prof8 + (size_t)(x >> 1) * Q.lp + r0) + (x & 1));
                if (BIAS) {
                    v.x = (int)__vadd4((uint32_t)v.x, b4); v.y = (int)__vadd4((uint32_t)v.y, b4);
                    v.z = (int)__vadd4((uint32_t)v.z, b4); v.w = (int)__vadd4((uint32_t)v.w, b4);
                }
                *reinterpret_cast<int4 *>(slice + (x >> 1) * SW16_ROW + (x & 1) * 16) = v;
            }
            __syncwarp();
            /* team: the previous pass (warp trank-1) must have published
             * column c before it is read */
            const long long in_base = (long long)((sp - 1) / tsize) * stride + 1;
            const long long out_base = (long long)(sp / tsize) * stride + 1;
            auto wait_for = [&](int c) -> bool {
                if (!team || sp == 0) return true;
                const int need = min(c, wmax - 1);
                bool ok = true;
                if (lane == 0 && need >= 0) {
                    const long long t0 = clock64();
                    while (s_prog[(trank + tsize - 1) % tsize] < in_base + need) {
                        if (*verr) { ok = false; break; }
                        if (clock64() - t0 > (1ll << 32)) { atomicExch(task_counter + 2, 1); ok = false; break; }
                    }
                    __threadfence_block();
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                __syncwarp();
                return ok;
            };
            /* columns [c0, c0 + 8) read the boundary up to column c0 + 11 */
            if (!wait_for(11)) break;
            uint32_t H[SW16_R], E[SW16_R];
#pragma unroll
            for (int r = 0; r < SW16_R; ++r) { H[r] = zeroH; E[r] = gapO; }
            uint32_t dg = zeroH;            /* lo: H(r0-1, j-1); hi: H(r0+15, j-2) */
            uint32_t prev_h = zeroH, prev_f = gapO;   /* lo halves: strip A bottom at j-1 */
            Sw16Best sa = {0, -1, -1}, sb = {0, -1, -1};
            /* what a column maximum has to pass (each half's own): the half's
             * best of this pass, and one less than the best of the other half
             * and of the passes before, whose equal in an earlier column
             * would win */
            uint32_t sbest = splat16(max(best.score - 1, 0) - bias);
            const bool more = r0 + 2 * SW16_R < ql;
            const int8_t *pb_at = slice + SW16_R;     /* strip B's scores of column j-1 */
            /* the pass boundary of a column is loaded four columns ahead: it
             * comes from L2 or DRAM, and the chain of one column is too short
             * to cover that latency (this pass overwrites entry j at column
             * j, never entry j+5). The first pass reads none: row -1 is H = 0,
             * F = -inf. */
            const uint32_t vnone = prmt(zeroH, gapO, 0x5410u);
            const int rd = r0 != 0 ? wmax : 0;
            uint32_t v_n[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v_n[k] = k < rd ? __ldcg(in_buf + (k + 1) * 32) : vnone;
            const uint32_t *in_at = in_buf + 5 * 32;
            uint32_t *out_at = out_buf;
            ResidueWords tw;
            tw.start(tseq, len);
            bool aborted = false;
            for (int j0 = 0; j0 <= wmax; j0 += 4, in_at += 4 * 32, out_at += 4 * 32) {
                if (team && j0 > 0 && (j0 & 7) == 0 && !wait_for(j0 + 11)) { aborted = true; break; }
                const uint32_t codes = tw.next(j0);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + u;
                    const uint32_t v = v_n[u];
                    v_n[u] = j + 4 < rd ? __ldcg(in_at + u * 32) : vnone;
                    uint32_t hu = prmt(v, prev_h, 0x5410u);     /* lo <- previous pass's strip B bottom */
                    uint32_t fu = prmt(v, prev_f, 0x5432u);
                    const int8_t *pa_at = slice + __byte_perm(codes, 0u, 0x4440u + u) * SW16_ROW;
                    const uint4 pa4 = *reinterpret_cast<const uint4 *>(pa_at);
                    const uint4 pb4 = *reinterpret_cast<const uint4 *>(pb_at);
                    pb_at = pa_at + SW16_R;
                    uint32_t hd = dg;
                    dg = hu;
                    uint32_t cmax = zeroH;
                    uint32_t aop = 0u;          /* BIAS: the previous row's max(H_diag + s, E, 0) - open */
#pragma unroll
                    for (int r = 0; r < SW16_R; ++r) {
                        const uint32_t wa = r < 4 ? pa4.x : r < 8 ? pa4.y : r < 12 ? pa4.z : pa4.w;
                        const uint32_t wb = r < 4 ? pb4.x : r < 8 ? pb4.y : r < 12 ? pb4.z : pb4.w;
                        uint32_t sc;
                        switch (r & 3) {
                            case 0: sc = pack_pair<0>(wa, wb); break;
                            case 1: sc = pack_pair<1>(wa, wb); break;
                            case 2: sc = pack_pair<2>(wa, wb); break;
                            default: sc = pack_pair<3>(wa, wb); break;
                        }
                        if (BIAS) {
                            /* registers hold HO = H - open and the profile s + open:
                             *   E(i,j) = max(E(i,j-1) - gap, HO(i,j-1))
                             *   a      = max(HO(i-1,j-1) + (s + open), E, 0)
                             *   F(i,j) = max(F(i-1,j) - gap, HO(i-1,j))
                             *          = max(F(i-1,j) - gap, a(i-1) - open)  (open >= gap)
                             *   HO     = max(a - open, F - open)
                             * so one DPX operation per row sits on the chain */
                            const uint32_t e = __viaddmax_s16x2(E[r], gapE, H[r]);
                            const uint32_t a = __viaddmax_s16x2_relu(hd, sc, e);
                            const uint32_t ao = __vadd2(a, gapO);
                            const uint32_t f = __viaddmax_s16x2(fu, gapE, r == 0 ? hu : aop);
                            const uint32_t ho = __viaddmax_s16x2(f, gapO, ao);
                            E[r] = e;
                            hd = H[r];
                            H[r] = ho;
                            hu = ho;
                            fu = f;
                            aop = ao;
                            if (r & 1) cmax = __vimax3_s16x2(cmax, H[r - 1], ho);
                        } else {
                            /* E(i,j) = max(E(i,j-1) - gap, H(i,j-1) - open): off the chain */
                            const uint32_t e = __viaddmax_s16x2(E[r], gapE, __vadd2(H[r], gapO));
                            const uint32_t a = __viaddmax_s16x2_relu(hd, sc, e);
                            /* F(i,j) = max(H(i-1,j) - open, F(i-1,j) - gap): on the chain */
                            const uint32_t f = __viaddmax_s16x2(hu, gapO, __vadd2(fu, gapE));
                            const uint32_t h = __vmaxs2(a, f);
                            E[r] = e;
                            hd = H[r];
                            H[r] = h;
                            hu = h;
                            fu = f;
                            if (r & 1) cmax = __vimax3_s16x2(cmax, H[r - 1], h);
                        }
                    }
                    if (more) out_at[u * 32] = prmt(hu, fu, 0x7632u);     /* column j - 1 */
                    prev_h = hu;
                    prev_f = fu;
                    if (u == 0 && j0 == 0) {
                        /* the high half computed column -1: restore strip B's
                         * left boundary (H = 0, E = -inf) */
#pragma unroll
                        for (int r = 0; r < SW16_R; ++r) {
                            H[r] = (H[r] & 0xffffu) | (zeroH & 0xffff0000u);
                            E[r] = (E[r] & 0xffffu) | (gapO & 0xffff0000u);
                        }
                    }
                    if (__vmaxs2(sbest, cmax) != sbest) {
                        const bool ge_lo = s16lo(cmax) <= s16lo(sbest), ge_hi = s16hi(cmax) <= s16hi(sbest);
                        /* past its half's bound: keep the column (the warp
                         * takes this branch whenever any lane does, so the row
                         * is looked up once per pass, from the saved column).
                         * Columns outside the target only raise the bound, and
                         * the high half's column -1 counts for nothing. */
                        int ba = s16lo(sbest), bb = s16hi(sbest);
                        if (!ge_lo) {
                            ba = s16lo(cmax);
                            if (j < len) {
#pragma unroll
                                for (int k = 0; k < SW16_R / 4; ++k)
                                    save[k] = make_uint4(H[4 * k], H[4 * k + 1], H[4 * k + 2], H[4 * k + 3]);
                                sa.score = ba + bias; sa.j = j;
                                bb = max(bb, ba - 1);
                            }
                        }
                        if (!ge_hi && j >= 1) {
                            const int c = s16hi(cmax);
                            bb = max(bb, c);
                            if (j <= len) {
#pragma unroll
                                for (int k = 0; k < SW16_R / 4; ++k)
                                    save[SW16_R / 4 + k] = make_uint4(H[4 * k], H[4 * k + 1], H[4 * k + 2], H[4 * k + 3]);
                                sb.score = c + bias; sb.j = j - 1;
                                ba = max(ba, c - 1);
                            }
                        }
                        sbest = (uint32_t)(uint16_t)ba | ((uint32_t)(uint16_t)bb << 16);
                    }
                }
                /* team: columns up to j0 + 2 are out */
                if (team && more && (j0 & 4)) {
                    __threadfence_block();
                    __syncwarp();
                    if (lane == 0) s_prog[trank] = out_base + min(j0 + 2, wmax - 1);
                }
            }
            if (team && more && !aborted) {
                __threadfence_block();
                __syncwarp();
                if (lane == 0) s_prog[trank] = out_base + wmax - 1;
            }
            if (aborted) break;
            /* the first row of each strip's best column reaching its maximum */
            if (sa.j >= 0) {
                int rr = SW16_R - 1;
#pragma unroll
                for (int k = SW16_R / 4 - 1; k >= 0; --k) {
                    const uint4 w = save[k];
                    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int x = 3; x >= 0; --x) if (s16lo(ws[x]) == sa.score - bias) rr = 4 * k + x;
                }
                sa.i = r0 + rr;
            }
            if (sb.j >= 0) {
                int rr = SW16_R - 1;
#pragma unroll
                for (int k = SW16_R / 4 - 1; k >= 0; --k) {
                    const uint4 w = save[SW16_R / 4 + k];
                    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int x = 3; x >= 0; --x) if (s16hi(ws[x]) == sb.score - bias) rr = 4 * k + x;
                }
                sb.i = r0 + SW16_R + rr;
            }
            fold_best(best, sa);
            fold_best(best, sb);
        }
        if (team) {
            /* merge the warps' per-lane bests: highest score, then smallest
             * column, then smallest row (the reference's first maximum) */
            s_best[wid][lane] = best;
            __syncthreads();
            if (wid != 0) continue;
            for (int w = 1; w < SW16_WARPS; ++w) {
                const Sw16Best c = s_best[w][lane];
                if (c.score > best.score || (c.score == best.score && (c.j < best.j ||
                                                                        (c.j == best.j && c.i < best.i))))
                    best = c;
            }
        }
        /* no positive cell: score 0 at (0, 0), the first cell (src/sw.c:150-158) */
        if (valid) {
            pb_pair_out o = {};
            o.score = best.score;
            o.end_query = best.i;
            o.end_ref = best.j;
            o.max_h = o.score;
            o.status = len != p.tlen[pid] ? PB_ST_OVERFLOW16 | PB_ST_BADCODE
                     : best.score >= Q.posmax ? PB_ST_OVERFLOW16 : 0;
            p.out[(size_t)T.q * p.npairs + pid] = o;
        }
    }
}

/*
 * Small searches and single pairs whose scores or penalties may pass 16 bits
 * (the others run on k_sw_wave16): the intra-task wavefront. One warp aligns one (query, target) pair in
 * exact int32: a pass covers 32 * RL query rows, RL per lane, and lane k
 * computes column t - k at iteration t, so the warp's 32 lanes work on 32
 * columns of one pair at once and the row-to-row dependency chain is RL
 * rows long instead of the inter-task kernel's per-target 16-row strips on
 * a handful of SMs. Row above a lane's first row: the previous lane's last
 * row by __shfl_up_sync, or, for lane 0, the previous pass's bottom row
 * from the warp's buffer (passes of one pair run one after the other on
 * the warp). The recurrence and end rule are src/sw.c:102-158's: H =
 * max(0, H_diag + s, E, F), the first maximum in column-major order, score
 * 0 at (0, 0) when no cell is positive; with open >= gap, F of the next
 * row is max(F - gap, max(a, 0) - open) with a = max(H_diag + s, E), one
 * dependent operation per row.
 */
/* RL query rows per lane (4, 8, 12 or 16; a pass covers 32 * RL rows),
 * chosen per launch from the query lengths (sw16_prepare) */
template <bool GE, int RL>
__global__ void __launch_bounds__(SW16_WARPS * 32, 2)
k_sw_wave(Sw16Params p, int *counter)
{
    extern __shared__ __align__(16) int8_t s_prof[];
    {
        const int4 *src = reinterpret_cast<const int4 *>(p.prof_all);
        int4 *dst = reinterpret_cast<int4 *>(s_prof);
        const int n16 = p.prof_bytes / 16;
        for (int k = threadIdx.x; k < n16; k += blockDim.x) dst[k] = src[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    int2 *buf = reinterpret_cast<int2 *>(p.scratch) + (size_t)(blockIdx.x * SW16_WARPS + wid) * p.maxlen;
    const int open = p.open, gap = p.gap;
    const int NEG = INT_MIN / 4;
    const long long nitems = (long long)p.nq * p.npairs;
    for (;;) {
        long long w = 0;
        if (lane == 0) w = atomicAdd(counter, 1);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= nitems) break;
        const int q = (int)(w / p.npairs);
        const int pid = p.order[w % p.npairs];
        const Sw16Query Q = p.queries[q];
        const int n = Q.qlen, m = p.tlen[pid];
        const uint8_t *ts = p.targets + p.toff[pid];
        const int8_t *prof = s_prof + Q.prof_off;
        const int npass = (n + 32 * RL - 1) / (32 * RL);
        Sw16Best best = {0, -1, -1};
        int status = 0;
        for (int pass = 0; pass < npass; ++pass) {
            const int R0 = pass * 32 * RL + lane * RL;
            /* a lane whose rows reach past lp (a multiple of 64, at least
             * qlen + 32) holds only dummy rows: they score 0 */
            const bool rows_in = R0 + RL <= Q.lp;
            int Hl[RL], E[RL];
#pragma unroll
            for (int r = 0; r < RL; ++r) { Hl[r] = 0; E[r] = NEG; }
            int dg = 0;                               /* H(R0 - 1, j - 1); H(i, -1) = 0 */
            int sh_h = 0, sh_f = NEG;
            int2 cur = make_int2(0, NEG);
            const int nreal = min(RL, max(0, n - R0));
            auto res_at = [&](int c) -> int { return (c >= 0 && c < m) ? (int)ts[c] : 0; };
            int tc_n1 = res_at(-lane), tc_n2 = res_at(1 - lane);
            for (int it = 0; it <= m - 1 + 31; ++it) {
                const int j = it - lane;
                if (((it & 31) == 0) && pass > 0) {
                    const int c = it + lane;
                    cur = c < m ? __ldcg(&buf[c]) : make_int2(0, NEG);
                }
                const int vh = __shfl_sync(0xffffffffu, cur.x, it & 31);
                const int vf = __shfl_sync(0xffffffffu, cur.y, it & 31);
                int up_h = __shfl_up_sync(0xffffffffu, sh_h, 1);
                int up_f = __shfl_up_sync(0xffffffffu, sh_f, 1);
                const int tc_raw = tc_n1;
                tc_n1 = tc_n2;
                tc_n2 = res_at(j + 2);
                if (lane == 0) {
                    /* row above the pass: row -1 (H = 0, F = -inf) or the
                     * previous pass's bottom row */
                    up_h = pass > 0 ? vh : 0;
                    up_f = pass > 0 ? vf : NEG;
                }
                if (j >= 0 && j < m) {
                    int tc = tc_raw;
                    if (tc >= p.nletters) { status |= PB_ST_BADCODE; tc = 0; }
                    /* R0 and lp are multiples of 4: word loads */
                    uint32_t sw[RL / 4];
#pragma unroll
                    for (int k = 0; k < RL / 4; ++k)
                        sw[k] = rows_in ? reinterpret_cast<const uint32_t *>(prof + (size_t)tc * Q.lp + R0)[k] : 0u;
                    int hd = dg;
                    int f = max(up_f - gap, up_h - open);
                    int cmax = 0, last_h = 0, last_f = 0;
#pragma unroll
                    for (int r = 0; r < RL; ++r) {
                        const int sc = (int)(int8_t)((sw[r >> 2] >> (8 * (r & 3))) & 0xffu);
                        const int e = max(E[r] - gap, Hl[r] - open);
                        const int a = __viaddmax_s32(hd, sc, e);
                        const int h = __vimax_s32_relu(a, f);
                        if (r < nreal) cmax = max(cmax, h);
                        last_h = h;
                        last_f = f;
                        if (GE) f = __viaddmax_s32(f, -gap, max(a, 0) - open);
                        else f = __viaddmax_s32(f, -gap, h - open);
                        E[r] = e;
                        hd = Hl[r];
                        Hl[r] = h;
                    }
                    /* a higher maximum than the lane's best, or the same one
                     * in an earlier column (a later pass revisits the
                     * columns): the first row reaching it in this column */
                    if (cmax > best.score || (cmax == best.score && j < best.j)) {
                        int rr = 0;
#pragma unroll
                        for (int r = RL - 1; r >= 0; --r) if (r < nreal && Hl[r] == cmax) rr = r;
                        best.score = cmax; best.j = j; best.i = R0 + rr;
                    }
                    dg = up_h;
                    sh_h = last_h;
                    sh_f = last_f;
                    if (lane == 31 && pass + 1 < npass) buf[j] = make_int2(last_h, last_f);
                }
            }
            __syncwarp();
        }
        /* the lanes' bests in the reference's order: higher score, then
         * smaller column, then smaller row */
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int os = __shfl_xor_sync(0xffffffffu, best.score, o);
            const int oj = __shfl_xor_sync(0xffffffffu, best.j, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best.i, o);
            const bool take = oj >= 0 && (best.j < 0 || os > best.score ||
                                          (os == best.score && (oj < best.j || (oj == best.j && oi < best.i))));
            if (take) { best.score = os; best.j = oj; best.i = oi; }
        }
        status = __reduce_or_sync(0xffffffffu, status);
        if (lane == 0) {
            pb_pair_out o = {};
            o.score = best.j >= 0 ? best.score : 0;
            o.end_query = best.j >= 0 ? best.i : 0;
            o.end_ref = best.j >= 0 ? best.j : 0;
            o.max_h = o.score;
            o.status = status;
            p.out[(size_t)q * p.npairs + pid] = o;
        }
    }
}

/*
 * The wavefront of small searches and single pairs in int16x2, where no
 * pair can leave 16 bits (the host's bound, wave16_ok): one warp per pair,
 * lane k holding 2R query rows as two strips of R rows in the halves of its
 * registers, strip B one column behind strip A as in k_sw16. Lane k works on
 * column t - 2k at iteration t (strip B on t - 2k - 1), so the row above its
 * strip A is lane k-1's strip B bottom of the iteration before: one shuffle
 * of (H, F) packed in a word.
 * What bounds it is the latency of one iteration -- the shuffle, R dependent
 * F steps, the hand-over -- with at most a few warps per scheduler, so the
 * rows per lane follow the query length (R = 5 for 300 rows: one pass), and
 * nothing is predicated: columns outside the target meet the letter after
 * the alphabet, whose scores of -128 leave the zero boundary before column 0
 * as it is and cannot raise a maximum after the last. Scores are staged per
 * block as [pass][letter][strip][lane], so that the lanes' loads fall on
 * different banks whatever their letters. One pair (300 x 350) takes 163 ->
 * 78.5 us per call, 1 query (300) x 1,000 targets 253 -> 107 us per plan run,
 * against the exact 32-bit wavefront (k_sw_wave), which stays for pairs that
 * may pass 16 bits. It runs up to a task per resident block (9,472 targets),
 * where it beats k_sw16 at 300 rows and more: 300 rows x 1,000 / 4,000 / 9,000
 * targets 107 / 172 / 324 us against 316 / 314 / 466 (9,600 targets), 800 rows x
 * 9,000 749 against 908, 1,500 rows 1,188 against 1,590. At 100 rows the two
 * are even there (214, 217); at 30 rows k_sw16 would be faster (185, 139).
 */
template <bool BIAS, int R>
__global__ void __launch_bounds__(WAVE16_WARPS * 32, 4)
k_sw_wave16(Sw16Params p, int *counter)
{
    constexpr int W = (R + 3) / 4;                 /* score words per strip */
    constexpr int LETTER = 2 * 32 * W;             /* words per letter */
    extern __shared__ __align__(16) uint32_t s_sc[];
    __shared__ int s_chunk;
    __shared__ uint16_t s_ring[WAVE16_WARPS][128];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    uint16_t *ring = s_ring[wid];
    const int L = p.nletters;
    uint32_t *buf = p.scratch + (size_t)(blockIdx.x * WAVE16_WARPS + wid) * p.maxlen;
    const uint32_t gapO = splat16(-p.open);
    const uint32_t gapE = splat16(-p.gap);
    const uint32_t zeroH = BIAS ? gapO : 0u;
    const int bias = BIAS ? p.open : 0;
    const uint32_t vnone = prmt(zeroH, gapO, 0x5410u);
    const int per_q = (p.npairs + WAVE16_WARPS - 1) / WAVE16_WARPS;
    const int nchunks = per_q * p.nq;
    int staged = -1;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_chunk = atomicAdd(counter, 1);
        __syncthreads();
        const int chunk = s_chunk;
        if (chunk >= nchunks) break;
        const int q = chunk / per_q;
        const Sw16Query Q = p.queries[q];
        const int n = Q.qlen;
        const int npass = (n + 64 * R - 1) / (64 * R);
        if (q != staged) {
            /* a thread stages one (strip, lane) of every second letter: R
             * bytes of the profile each, + open in the biased form */
            const int slot = threadIdx.x & 63;
            for (int pass = 0; pass < npass; ++pass) {
                const int row = (pass * 32 + (slot & 31)) * 2 * R + (slot >> 5) * R;
                uint32_t *d = s_sc + (size_t)pass * (L + 1) * LETTER + (slot >> 5) * 32 * W + (slot & 31) * W;
#pragma unroll 4
                for (int a = threadIdx.x >> 6; a <= L; a += WAVE16_WARPS / 2) {
                    uint32_t w[W];
#pragma unroll
                    for (int k = 0; k < W; ++k) w[k] = 0u;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        int v = -128;
                        if (a < L) v = (row + r < Q.lp ? (int)__ldg(Q.prof8 + (size_t)a * Q.lp + row + r) : 0) + bias;
                        w[r >> 2] |= (uint32_t)(uint8_t)(int8_t)v << (8 * (r & 3));
                    }
#pragma unroll
                    for (int k = 0; k < W; ++k) d[(size_t)a * LETTER + k] = w[k];
                }
            }
            staged = q;
            __syncthreads();
        }
        const int item = (chunk - q * per_q) * WAVE16_WARPS + wid;
        if (item >= p.npairs) continue;
        const int pid = p.order[item];
        const int m = p.tlen[pid];
        const uint8_t *ts = p.targets + p.toff[pid];
        Sw16Best best = {0, 0, 0};
        int status = 0;
        for (int pass = 0; pass < npass; ++pass) {
            const uint32_t *sc_pass = s_sc + (size_t)pass * (L + 1) * LETTER + lane * W;
            const int R0 = (pass * 32 + lane) * 2 * R;
            const bool more = pass + 1 < npass;
            uint32_t H[R], E[R];
#pragma unroll
            for (int r = 0; r < R; ++r) { H[r] = zeroH; E[r] = gapO; }
            uint32_t dg = zeroH, prev_h = zeroH, prev_f = gapO, cur = vnone;
            /* as in k_sw16: a half's own best of this pass, and one less than
             * any other known score (every 32 columns, the warp's) */
            uint32_t sbest = splat16(max(best.score - 1, 0) - bias);
            Sw16Best sa = {0, -1, -1}, sb = {0, -1, -1};
            uint32_t SA[R], SB[R];                 /* the strips' best columns */
#pragma unroll
            for (int r = 0; r < R; ++r) { SA[r] = 0u; SB[r] = 0u; }
            /* Letters by column in the warp's ring of four 32-column chunks, as
             * word offsets of their scores: a chunk is checked and stored once
             * by the whole warp, one chunk before lane 0 needs it (a load per
             * lane and column waited for its check in every iteration). */
            auto fetch = [&](int c) -> int { return c < m ? (int)__ldg(ts + c) : L; };
            auto put = [&](int c, int v) {
                if (c < m && v >= L) { v = 0; status |= PB_ST_BADCODE; }
                ring[c & 127] = (uint16_t)(v * LETTER);
            };
            __syncwarp();
            put(lane, fetch(lane));
            ring[64 + lane] = ring[96 + lane] = (uint16_t)(L * LETTER);
            int pre = fetch(32 + lane);
            __syncwarp();
            /* A column's scores are loaded, and the row above handed down,
             * right when the column before allows it, before that column's
             * check for a new best: issue is in order, and a branch between
             * would add its latency to the chain. */
            auto load = [&](uint32_t (&w)[W], const uint32_t *at) {
                if (W == 2) {
                    const uint2 x = *reinterpret_cast<const uint2 *>(at);
                    w[0] = x.x; w[W - 1] = x.y;
                } else {
                    w[0] = *at;
                }
            };
            const uint32_t *pa_at = sc_pass + (lane == 0 ? ring[0] : L * LETTER);
            uint32_t wa[W], wb4[W], v = vnone;
            load(wa, pa_at);
            load(wb4, sc_pass + L * LETTER + 32 * W);
            const int iters = m + 63;
            for (int t0 = 0; t0 < iters; t0 += 32) {
                if (pass > 0) {
                    cur = t0 + lane < m ? __ldcg(&buf[t0 + lane]) : vnone;
                    const uint32_t vin = __shfl_sync(0xffffffffu, cur, 0);
                    if (lane == 0) v = vin;
                }
                put(t0 + 32 + lane, pre);
                pre = fetch(t0 + 64 + lane);
                const int wb = __reduce_max_sync(0xffffffffu, max(best.score, max(sa.score, sb.score)));
                sbest = __vmaxs2(sbest, splat16(max(wb - 1, 0) - bias));
                __syncwarp();
                const int n_it = min(32, iters - t0);
                /* strip A's column j = t0 + it - 2 * lane */
                int off = ring[(t0 - 2 * lane + 1) & 127];
#pragma unroll 2
                for (int it = 0; it < n_it; ++it) {
                    const int j = t0 + it - 2 * lane;
                    uint32_t na[W], nb[W];
                    load(nb, pa_at + 32 * W);
                    pa_at = sc_pass + off;
                    load(na, pa_at);
                    off = ring[(j + 2) & 127];
                    uint32_t hu = prmt(v, prev_h, 0x5410u);
                    uint32_t fu = prmt(v, prev_f, 0x5432u);
                    uint32_t hd = dg;
                    dg = hu;
                    uint32_t cmax = zeroH, aop = 0u;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        uint32_t sc;
                        switch (r & 3) {
                            case 0: sc = pack_pair<0>(wa[r >> 2], wb4[r >> 2]); break;
                            case 1: sc = pack_pair<1>(wa[r >> 2], wb4[r >> 2]); break;
                            case 2: sc = pack_pair<2>(wa[r >> 2], wb4[r >> 2]); break;
                            default: sc = pack_pair<3>(wa[r >> 2], wb4[r >> 2]); break;
                        }
                        uint32_t e, a, f, h;
                        if (BIAS) {
                            e = __viaddmax_s16x2(E[r], gapE, H[r]);
                            a = __viaddmax_s16x2_relu(hd, sc, e);
                            const uint32_t ao = __vadd2(a, gapO);
                            f = __viaddmax_s16x2(fu, gapE, r == 0 ? hu : aop);
                            h = __viaddmax_s16x2(f, gapO, ao);
                            aop = ao;
                        } else {
                            e = __viaddmax_s16x2(E[r], gapE, __vadd2(H[r], gapO));
                            a = __viaddmax_s16x2_relu(hd, sc, e);
                            f = __viaddmax_s16x2(hu, gapO, __vadd2(fu, gapE));
                            h = __vmaxs2(a, f);
                        }
                        E[r] = e;
                        hd = H[r];
                        H[r] = h;
                        hu = h;
                        fu = f;
                        if (r & 1) cmax = __vimax3_s16x2(cmax, H[r - 1], h);
                        else if (r == R - 1) cmax = __vmaxs2(cmax, h);
                    }
                    const uint32_t out = prmt(hu, fu, 0x7632u);
                    v = __shfl_up_sync(0xffffffffu, out, 1);
                    const uint32_t vin = pass > 0 ? __shfl_sync(0xffffffffu, cur, (it + 1) & 31) : vnone;
                    if (lane == 0) v = vin;
                    prev_h = hu;
                    prev_f = fu;
#pragma unroll
                    for (int k = 0; k < W; ++k) { wa[k] = na[k]; wb4[k] = nb[k]; }
                    if (more && lane == 31 && (unsigned)(j - 1) < (unsigned)m) buf[j - 1] = out;
                    if (__vmaxs2(sbest, cmax) != sbest) {
                        const int ca = s16lo(cmax), cb = s16hi(cmax);
                        int ba = s16lo(sbest), bb = s16hi(sbest);
                        const bool up_a = ca > ba, up_b = cb > bb;
                        if (up_a) {
#pragma unroll
                            for (int r = 0; r < R; ++r) SA[r] = H[r];
                            sa.score = ca + bias; sa.j = j;
                            ba = ca;
                        }
                        if (up_b) {
#pragma unroll
                            for (int r = 0; r < R; ++r) SB[r] = H[r];
                            sb.score = cb + bias; sb.j = j - 1;
                            bb = cb;
                        }
                        if (up_a) bb = max(bb, ca - 1);
                        if (up_b) ba = max(ba, cb - 1);
                        sbest = (uint32_t)(uint16_t)ba | ((uint32_t)(uint16_t)bb << 16);
                    }
                }
            }
            /* the first row of each strip's best column reaching its maximum */
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const Sw16Best c = h ? sb : sa;
                if (c.j < 0) continue;
                int rr = R - 1;
#pragma unroll
                for (int r = R - 2; r >= 0; --r) if ((h ? s16hi(SB[r]) : s16lo(SA[r])) == c.score - bias) rr = r;
                const int ci = R0 + h * R + rr;
                if (c.score > best.score || (c.score == best.score && (c.j < best.j || (c.j == best.j && ci < best.i)))) {
                    best.score = c.score; best.j = c.j; best.i = ci;
                }
            }
            __syncwarp();
        }
        /* the lanes' bests in the reference's order: higher score, then
         * smaller column, then smaller row */
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int os = __shfl_xor_sync(0xffffffffu, best.score, o);
            const int oj = __shfl_xor_sync(0xffffffffu, best.j, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best.i, o);
            if (os > best.score || (os == best.score && (oj < best.j || (oj == best.j && oi < best.i)))) {
                best.score = os; best.j = oj; best.i = oi;
            }
        }
        status = __reduce_or_sync(0xffffffffu, status);
        if (lane == 0) {
            pb_pair_out o = {};
            o.score = best.score;
            o.end_query = best.i;
            o.end_ref = best.j;
            o.max_h = o.score;
            o.status = status;
            p.out[(size_t)q * p.npairs + pid] = o;
        }
    }
}

}  // namespace pb

namespace {

__global__ void k_iota(int *v, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

__global__ void k_collect_overflow(const pb_pair_out *out, int n, int *list, int *count,
                                   const int64_t *toff, const int *tlen,
                                   int64_t *otoff, int *otlen)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && (out[i].status & PB_ST_OVERFLOW16)) {
        const int k = atomicAdd(count, 1);
        list[k] = i;
        otoff[k] = toff[i];
        otlen[k] = tlen[i];
    }
}

__global__ void k_count_overflow(const pb_pair_out *__restrict__ out, size_t n, int *__restrict__ count)
{
    int c = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        c += (out[i].status & PB_ST_OVERFLOW16) != 0;
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

__global__ void k_scatter(const pb_pair_out *src, const int *list, int n, pb_pair_out *dst)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[list[k]] = src[k];
}

}  // namespace

/* the largest profiles, or staged scores, that the kernels of small searches
 * take into shared memory; also the documented limit of a plan's profiles */
static constexpr size_t SW16_WAVE_SMEM = 200 * 1024;

/* Everything the score kernel needs for a batch that depends only on the
 * profiles and the target lengths: the task list (most cells first, team
 * tasks at the front), the concatenated int8 profiles and the sizes of the
 * per-warp pass buffers. Buffers come from st's pool
 * and are released by sw16_release. */
struct Sw16Prep {
    pb::Sw16Params p;
    int blocks;
    bool wave;                    /* few tasks: the intra-task wavefront k_sw_wave */
    int wave_rl;                  /* its rows per lane */
    int wave16;                   /* > 0: k_sw_wave16 with that many rows per strip instead */
    size_t smem;                  /* dynamic shared memory of its kernel */
    int *counter;                 /* [warp tasks, team tasks, error, spare] */
    size_t scratch_bytes, colsave_bytes;
    void *bufs[4];
};

static void sw16_release(Sw16Prep *pr, cudaStream_t st)
{
    for (void *x : pr->bufs) if (x) cudaFreeAsync(x, st);
    memset(pr->bufs, 0, sizeof pr->bufs);
}

typedef void (*WaveKernel)(pb::Sw16Params, int *);

/* k_sw_wave for (open >= gap, rows per lane) */
static WaveKernel wave_kernel(bool ge, int rl)
{
    if (ge) {
        switch (rl) {
            case 4: return pb::k_sw_wave<true, 4>;
            case 12: return pb::k_sw_wave<true, 12>;
            case 16: return pb::k_sw_wave<true, 16>;
            default: return pb::k_sw_wave<true, 8>;
        }
    }
    switch (rl) {
        case 4: return pb::k_sw_wave<false, 4>;
        case 12: return pb::k_sw_wave<false, 12>;
        case 16: return pb::k_sw_wave<false, 16>;
        default: return pb::k_sw_wave<false, 8>;
    }
}

/* k_sw_wave16 for (biased, rows per strip) */
template <bool BIAS>
static WaveKernel wave16_kernel_of(int r)
{
    switch (r) {
        case 1: return pb::k_sw_wave16<BIAS, 1>;
        case 2: return pb::k_sw_wave16<BIAS, 2>;
        case 3: return pb::k_sw_wave16<BIAS, 3>;
        case 4: return pb::k_sw_wave16<BIAS, 4>;
        case 5: return pb::k_sw_wave16<BIAS, 5>;
        case 6: return pb::k_sw_wave16<BIAS, 6>;
        case 7: return pb::k_sw_wave16<BIAS, 7>;
        default: return pb::k_sw_wave16<BIAS, 8>;
    }
}

static WaveKernel wave16_kernel(bool bias, int r) { return bias ? wave16_kernel_of<true>(r) : wave16_kernel_of<false>(r); }

/* every score + open inside int8, open >= gap: the biased kernels */
static bool sw16_bias_ok(const pb_device_profile *dp, int open, int gap)
{
    return open >= gap && dp->mmax + open <= 127 && dp->mmin + open >= -128;
}

/* Can no pair of this profile with a target of at most maxlen residues leave
 * k_sw_wave16's lanes? Every H is at most max(matrix) per aligned pair (below
 * the same bound as k_sw16's overflow check), and E, F are at least -open -
 * gap. */
static bool wave16_ok(const pb_device_profile *dp, int maxlen, int open, int gap)
{
    const long long top = (long long)std::max(dp->mmax, 0) * (std::min(dp->qlen, maxlen) + 1);
    return dp->fits8 && open + gap <= 30000 && top < 32767 - std::max(dp->mmax, 0) - 1;
}

/* rows per strip: the fewest row-steps over the queries, npass * (R + 3) per
 * column, the 3 standing for an iteration's shuffles, loads and checks */
static int wave16_rows(const pb_device_profile *const *profs, int nq)
{
    int best_r = 8;
    double best = -1.0;
    for (int r = 1; r <= 8; ++r) {
        double cost = 0.0;
        for (int q = 0; q < nq; ++q) cost += (double)((profs[q]->qlen + 64 * r - 1) / (64 * r)) * (r + 3);
        if (best < 0.0 || cost < best) { best = cost; best_r = r; }
    }
    return best_r;
}

/* bytes of one query's staged scores */
static size_t wave16_smem(const pb_device_profile *dp, int r)
{
    return (size_t)((dp->qlen + 64 * r - 1) / (64 * r)) * (dp->size + 1) * 64 * 4 * ((r + 3) / 4);
}

static void wave_set_smem(int bytes)
{
    for (int ge = 0; ge < 2; ++ge)
        for (int rl = 4; rl <= 16; rl += 4)
            pb_raise_smem((const void *)wave_kernel(ge != 0, rl), bytes);
}

/* The length order of a batch's targets, shared by the launches of one
 * search: targets by descending length (device), their lengths (host). */
struct Sw16Sort {
    int *order = nullptr;
    std::vector<int> hlen;
    void *bufs[4] = {nullptr, nullptr, nullptr, nullptr};
};

static void sw16_sort_release(Sw16Sort *so, cudaStream_t st)
{
    for (void *&x : so->bufs) { if (x) cudaFreeAsync(x, st); x = nullptr; }
}

/* synchronises st */
static int sw16_sort(const pb_batch *b, cudaStream_t st, Sw16Sort *so)
{
    const int n = b->npairs;
    int *keys_sorted = nullptr, *idx = nullptr, *order = nullptr;
    void *tmp = nullptr;
    size_t tmp_sort = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp_sort, b->d_tlen, keys_sorted, idx, order, n, 0, 32, st);
    /* an allocation that fails ends the call before anything writes
     * through it, releasing what was allocated */
    if (cudaMallocAsync((void **)&keys_sorted, sizeof(int) * n, st) == cudaSuccess) so->bufs[0] = keys_sorted;
    if (cudaMallocAsync((void **)&idx, sizeof(int) * n, st) == cudaSuccess) so->bufs[1] = idx;
    if (cudaMallocAsync((void **)&order, sizeof(int) * n, st) == cudaSuccess) so->bufs[2] = order;
    if (cudaMallocAsync(&tmp, tmp_sort, st) == cudaSuccess) so->bufs[3] = tmp;
    for (void *x : so->bufs)
        if (!x) {
            sw16_sort_release(so, st);
            cudaGetLastError();
            return -1;
        }
    so->order = order;
    k_iota<<<(n + 255) / 256, 256, 0, st>>>(idx, n);
    cub::DeviceRadixSort::SortPairsDescending(tmp, tmp_sort, b->d_tlen, keys_sorted, idx, order, n, 0, 32, st);
    so->hlen.resize(n);
    cudaMemcpyAsync(so->hlen.data(), keys_sorted, sizeof(int) * n, cudaMemcpyDeviceToHost, st);
    return cudaStreamSynchronize(st) == cudaSuccess ? 0 : -1;
}

/* b's profiles against its targets in the order of `so` (which outlives the
 * launch) */
static int sw16_prepare(const pb_batch *b, pb_pair_out *d_out_all, const Sw16Sort &so, cudaStream_t st, Sw16Prep *pr)
{
    const int n = b->npairs, nq = b->nprofs;
    memset(pr, 0, sizeof *pr);
    const std::vector<int> &hlen = so.hlen;
    int *counter = nullptr;
    int8_t *prof_all = nullptr;
    pb::Sw16Task *d_tasks = nullptr;
    pb::Sw16Query *d_q = nullptr;
    /* an allocation that fails ends the call before anything writes
     * through it, releasing what was allocated */
    auto give_up = [&]() {
        void *owned[4] = {counter, prof_all, d_tasks, d_q};
        memcpy(pr->bufs, owned, sizeof owned);
        sw16_release(pr, st);
        cudaGetLastError();
        return -1;
    };
    int nsm = 0, dev = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    /* the biased kernel (one DPX operation per row on the dependency
     * chain) needs open >= gap and every score + open inside int8 */
    bool bias = b->open >= b->gap;
    size_t prof_bytes = 0;
    for (int q = 0; q < nq; ++q) {
        bias = bias && sw16_bias_ok(b->profs[q], b->open, b->gap);
        prof_bytes += (size_t)b->profs[q]->size * b->profs[q]->lp;
    }
    pr->smem = (size_t)pb::SW16_WARPS * b->profs[0]->size * pb::SW16_ROW;
    const void *kern = bias ? (const void *)pb::k_sw16<true> : (const void *)pb::k_sw16<false>;
    pb_raise_smem(kern, (int)pr->smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, pb::SW16_WARPS * 32, pr->smem);
    if (per_sm < 1) per_sm = 1;
    int blocks = per_sm * nsm;
    const int nblk = (n + 31) / 32;
    const size_t ntasks = (size_t)nq * nblk;
    /* few tasks (a small database, e.g. one query against 1,000 targets)
     * whose profiles fit its shared memory: the intra-task wavefront, a warp
     * per pair, as many warps as pairs (up to the resident warps) */
    int wave16 = wave16_rows(b->profs, nq);
    size_t smem16 = 0;
    for (int q = 0; q < nq; ++q) {
        if (!wave16_ok(b->profs[q], hlen[0], b->open, b->gap)) wave16 = 0;
        if (wave16) smem16 = std::max(smem16, wave16_smem(b->profs[q], wave16));
    }
    if (smem16 > SW16_WAVE_SMEM) wave16 = 0;
    const bool few = ntasks <= (size_t)blocks && (wave16 || prof_bytes <= SW16_WAVE_SMEM);
    if ((size_t)blocks > ntasks) blocks = (int)ntasks;
    pr->wave = few;
    /* the queries; for the wavefront their profiles side by side */
    std::vector<pb::Sw16Query> hq(nq);
    if (few && !wave16 && cudaMallocAsync((void **)&prof_all, prof_bytes, st) != cudaSuccess) return give_up();
    {
        size_t off = 0;
        for (int q = 0; q < nq; ++q) {
            const pb_device_profile *dp = b->profs[q];
            const size_t bytes = (size_t)dp->size * dp->lp;
            if (few && !wave16) cudaMemcpyAsync(prof_all + off, dp->d_prof8, bytes, cudaMemcpyDeviceToDevice, st);
            hq[q].prof8 = dp->d_prof8;
            hq[q].prof_off = few && !wave16 ? (int)off : 0;
            hq[q].qlen = dp->qlen;
            hq[q].lp = dp->lp;
            hq[q].posmax = 32767 - dp->mmax - 1;
            off += bytes;
        }
    }
    /* tasks: (query, block of 32 sorted targets), most columns (passes x
     * target length) first: every query's are in that order already, so the
     * queries' lists are merged */
    std::vector<pb::Sw16Task> tasks;
    std::vector<int64_t> cost;
    tasks.reserve(ntasks);
    cost.reserve(ntasks);
    {
        typedef std::pair<int64_t, int> Head;                 /* cost, query */
        std::vector<Head> heap;
        std::vector<int> at(nq, 0);
        auto cost_of = [&](int q, int k) {
            return (int64_t)((hq[q].qlen + 2 * pb::SW16_R - 1) / (2 * pb::SW16_R)) * (hlen[32 * (size_t)k] + 1);
        };
        for (int q = 0; q < nq; ++q) heap.push_back(Head(cost_of(q, 0), q));
        std::make_heap(heap.begin(), heap.end());
        while (!heap.empty()) {
            std::pop_heap(heap.begin(), heap.end());
            const Head h = heap.back();
            heap.pop_back();
            pb::Sw16Task t;
            t.q = h.second;
            t.first = 32 * at[h.second]++;
            tasks.push_back(t);
            cost.push_back(h.first);
            if (at[h.second] < nblk) {
                heap.push_back(Head(cost_of(h.second, at[h.second]), h.second));
                std::push_heap(heap.begin(), heap.end());
            }
        }
    }
    /* Team tasks, listed first: those that would hold up the end of the
     * launch on one warp. The warp tasks that follow end at most one task
     * after their fair share of the remaining work; a task above half of
     * that share therefore goes to a team (above the whole share where its
     * passes, fewer than a multiple of the team, would leave warps idle). */
    int nteam = 0;
    if (!few) {
        double rest = 0.0;
        for (int64_t c : cost) rest += (double)c;
        const double warps = (double)blocks * pb::SW16_WARPS;
        std::vector<pb::Sw16Task> lone;
        lone.reserve(ntasks);
        for (size_t k = 0; k < ntasks; ++k) {
            const int np = (hq[tasks[k].q].qlen + 2 * pb::SW16_R - 1) / (2 * pb::SW16_R);
            const int rounds = (np + pb::SW16_WARPS - 1) / pb::SW16_WARPS;
            const double part = np >= 0.7 * rounds * pb::SW16_WARPS ? 0.5 : 1.0;
            if (np > 1 && (double)cost[k] > part * rest / warps) {
                rest -= (double)cost[k];
                tasks[nteam++] = tasks[k];
            } else {
                lone.push_back(tasks[k]);
            }
        }
        std::copy(lone.begin(), lone.end(), tasks.begin() + nteam);
    }
    if (cudaMallocAsync((void **)&counter, sizeof(int) * 4, st) != cudaSuccess ||
        cudaMallocAsync((void **)&d_tasks, sizeof(pb::Sw16Task) * ntasks, st) != cudaSuccess ||
        cudaMallocAsync((void **)&d_q, sizeof(pb::Sw16Query) * nq, st) != cudaSuccess)
        return give_up();
    cudaMemsetAsync(counter, 0, sizeof(int) * 4, st);   /* warp tasks, team tasks, error */
    cudaMemcpyAsync(d_tasks, tasks.data(), sizeof(pb::Sw16Task) * ntasks, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_q, hq.data(), sizeof(pb::Sw16Query) * nq, cudaMemcpyHostToDevice, st);
    /* entry c + 1 of a pass buffer is column c; a pass writes up to four
     * past the longest target */
    const int maxlen = hlen[0] + 8;
    if (few && wave16) {
        pr->wave16 = wave16;
        pr->smem = smem16;
        const WaveKernel k16 = wave16_kernel(bias, wave16);
        int wper = 0;
        pb_raise_smem((const void *)k16, (int)smem16);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&wper, k16, pb::WAVE16_WARPS * 32, smem16);
        if (wper < 1) wper = 1;
        const long long want = (long long)nq * ((n + pb::WAVE16_WARPS - 1) / pb::WAVE16_WARPS);
        blocks = (int)std::min<long long>(want, (long long)wper * nsm);
    } else if (few) {
        /* rows per lane: the fewest row-steps over the batch's queries,
         * npass * (RL + 4) per column, the 4 standing for the per-column
         * shuffles and loads (one query of 300 rows: one pass of 12 rows
         * per lane instead of two of 8) */
        int best_rl = 8;
        double best_cost = -1.0;
        for (int rl = 4; rl <= 16; rl += 4) {
            double cost = 0.0;
            for (int q = 0; q < nq; ++q) cost += (double)((hq[q].qlen + 32 * rl - 1) / (32 * rl)) * (rl + 4);
            if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best_rl = rl; }
        }
        pr->wave_rl = best_rl;
        int wper = 0;
        pr->smem = prof_bytes;
        wave_set_smem((int)prof_bytes);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&wper, wave_kernel(b->open >= b->gap, best_rl),
                                                      pb::SW16_WARPS * 32, prof_bytes);
        if (wper < 1) wper = 1;
        const long long items = (long long)n * nq;
        const long long want = (items + pb::SW16_WARPS - 1) / pb::SW16_WARPS;
        blocks = (int)std::min<long long>(want, (long long)wper * nsm);
    }
    pr->scratch_bytes = few ? sizeof(int2) * (size_t)maxlen * blocks * pb::SW16_WARPS
                            : sizeof(uint32_t) * (size_t)maxlen * 32 * blocks * pb::SW16_WARPS;
    /* k_sw16: per thread, the two strips' best columns (2 x 16 words) */
    pr->colsave_bytes = few ? 0 : sizeof(uint4) * (pb::SW16_R / 2) * (size_t)blocks * pb::SW16_WARPS * 32;
    pb::Sw16Params &p = pr->p;
    p.open = b->open; p.gap = b->gap; p.npairs = n; p.nq = nq; p.nletters = b->profs[0]->size;
    p.bias = bias ? 1 : 0;
    p.ntasks = (int)ntasks; p.maxlen = maxlen; p.nteam = nteam;
    p.queries = d_q; p.prof_all = prof_all; p.prof_bytes = (int)prof_bytes;
    p.order = so.order; p.tasks = d_tasks;
    p.targets = b->d_targets; p.toff = b->d_toff; p.tlen = b->d_tlen;
    p.scratch = nullptr; p.colsave = nullptr;      /* sw16_workspace */
    p.out = d_out_all;
    pr->blocks = blocks;
    pr->counter = counter;
    void *owned[4] = {counter, prof_all, d_tasks, d_q};
    memcpy(pr->bufs, owned, sizeof owned);
    if (cudaGetLastError() != cudaSuccess) {
        sw16_release(pr, st);
        return -1;
    }
    return 0;
}

/* The pass buffers of a prepared batch. */
struct Sw16Work {
    uint32_t *scratch = nullptr;
    uint4 *colsave = nullptr;
};

static void sw16_work_release(Sw16Work *w, cudaStream_t st)
{
    if (w->scratch) cudaFreeAsync(w->scratch, st);
    if (w->colsave) cudaFreeAsync(w->colsave, st);
    w->scratch = nullptr;
    w->colsave = nullptr;
}

static int sw16_workspace(Sw16Prep *pr, cudaStream_t st, Sw16Work *w)
{
    if (cudaMallocAsync((void **)&w->scratch, pr->scratch_bytes, st) != cudaSuccess) w->scratch = nullptr;
    if (pr->colsave_bytes && cudaMallocAsync((void **)&w->colsave, pr->colsave_bytes, st) != cudaSuccess)
        w->colsave = nullptr;
    pr->p.scratch = w->scratch;
    pr->p.colsave = w->colsave;
    if (w->scratch && (w->colsave || !pr->colsave_bytes)) return 0;
    cudaGetLastError();
    return -1;
}

/* the kernel on a prepared batch (its counters zeroed first) */
static void sw16_launch(const Sw16Prep &pr, cudaStream_t st)
{
    cudaMemsetAsync(pr.counter, 0, sizeof(int) * 4, st);
    if (pr.wave16) {
        wave16_kernel(pr.p.bias != 0, pr.wave16)<<<pr.blocks, pb::WAVE16_WARPS * 32, pr.smem, st>>>(pr.p, pr.counter);
    } else if (pr.wave) {
        wave_kernel(pr.p.open >= pr.p.gap, pr.wave_rl)<<<pr.blocks, pb::SW16_WARPS * 32, pr.smem, st>>>(
            pr.p, pr.counter);
    } else {
        if (pr.p.bias)
            pb::k_sw16<true><<<pr.blocks, pb::SW16_WARPS * 32, pr.smem, st>>>(pr.p, pr.counter);
        else
            pb::k_sw16<false><<<pr.blocks, pb::SW16_WARPS * 32, pr.smem, st>>>(pr.p, pr.counter);
    }
}

/* nq profiles against the same targets; out[q * npairs + i]: one launch for
 * every query. */
extern "C" int pb_cuda_align_sw16_multi(const pb_batch *b, pb_pair_out *d_out_all)
{
    if (pb_cuda_init() != 0) return -1;
    const int n = b->npairs, nq = b->nprofs;
    if (n <= 0 || nq <= 0) return 0;
    bool ok = b->alg == PB_SW && !b->stats && !b->d_qlim && !b->d_tlim && b->open + b->gap <= 30000;
    for (int q = 0; q < nq && ok; ++q) ok = b->profs[q]->fits8 && b->profs[q]->size == b->profs[0]->size;
    if (!ok) {
        /* outside this kernel's domain: the exact kernel, one profile at a time */
        for (int q = 0; q < nq; ++q) {
            pb_batch one = *b;
            one.profs = &b->profs[q];
            one.nprofs = 1;
            one.d_out = d_out_all + (size_t)q * n;
            if (pb_cuda_align_exact(&one) != 0) return -1;
        }
        return 0;
    }
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return -1;
    Sw16Sort sort;
    Sw16Prep prep;
    Sw16Work work;
    memset(&prep, 0, sizeof prep);
    int rc = sw16_sort(b, st, &sort);
    if (rc == 0) rc = sw16_prepare(b, d_out_all, sort, st, &prep);
    if (rc == 0) rc = sw16_workspace(&prep, st, &work);
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    if (rc == 0 && (cudaEventCreate(&ev0) != cudaSuccess || cudaEventCreate(&ev1) != cudaSuccess)) rc = -1;
    if (rc == 0) {
        cudaEventRecord(ev0, st);
        sw16_launch(prep, st);
        cudaEventRecord(ev1, st);
        if (cudaGetLastError() != cudaSuccess) rc = -1;
        pb_diag_count_launch(2);   /* k_iota, the score kernel */
    }
    /* the launch's error flag, and the pairs that left the 16-bit range */
    int herr = 0, nover_all = 0;
    int *over = nullptr;
    const size_t N = (size_t)n * nq;
    if (rc == 0 && cudaMallocAsync((void **)&over, sizeof(int), st) != cudaSuccess) rc = -1;
    if (rc == 0) {
        cudaMemsetAsync(over, 0, sizeof(int), st);
        k_count_overflow<<<148, 256, 0, st>>>(d_out_all, N, over);
        pb_diag_count_launch(1);
        cudaMemcpyAsync(&nover_all, over, sizeof(int), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(&herr, prep.counter + 2, sizeof(int), cudaMemcpyDeviceToHost, st);
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
    if (herr) {
        fprintf(stderr, "pb_cuda_align_sw16_multi: a pass wait exceeded its bound\n");
        rc = -1;
    }
    if (rc == 0) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ev0, ev1);
        pb_diag_sw16_time(ms);
    }
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    /* pairs that left the 16-bit range: the exact kernel, per query */
    int *list = nullptr, *otlen = nullptr;
    int64_t *otoff = nullptr;
    if (rc == 0 && nover_all > 0 &&
        (cudaMallocAsync((void **)&list, sizeof(int) * n, st) != cudaSuccess ||
         cudaMallocAsync((void **)&otlen, sizeof(int) * n, st) != cudaSuccess ||
         cudaMallocAsync((void **)&otoff, sizeof(int64_t) * n, st) != cudaSuccess)) {
        cudaGetLastError();
        rc = -1;   /* nothing below runs; the buffers that exist are freed */
    }
    for (int q = 0; q < nq && rc == 0 && nover_all > 0; ++q) {
        int nover = 0;
        pb_pair_out *oq = d_out_all + (size_t)q * n;
        cudaMemsetAsync(over, 0, sizeof(int), st);
        k_collect_overflow<<<(n + 255) / 256, 256, 0, st>>>(oq, n, list, over, b->d_toff,
                                                            b->d_tlen, otoff, otlen);
        pb_diag_count_launch(1);
        cudaMemcpyAsync(&nover, over, sizeof(int), cudaMemcpyDeviceToHost, st);
        cudaStreamSynchronize(st);
        if (nover > 0) {
            pb_pair_out *tmpo = nullptr;
            if (cudaMallocAsync((void **)&tmpo, sizeof(pb_pair_out) * nover, st) != cudaSuccess) {
                cudaGetLastError();
                rc = -1;
                break;
            }
            cudaStreamSynchronize(st);
            pb_batch sub = *b;
            sub.profs = &b->profs[q];
            sub.nprofs = 1;
            sub.npairs = nover;
            sub.d_toff = otoff;
            sub.d_tlen = otlen;
            sub.d_out = tmpo;
            sub.d_prof_index = nullptr;
            rc = pb_cuda_align_exact(&sub);
            k_scatter<<<(nover + 255) / 256, 256, 0, st>>>(tmpo, list, nover, oq);
            pb_diag_count_launch(1);
            cudaFreeAsync(tmpo, st);
        }
    }
    if (list) cudaFreeAsync(list, st);
    if (otlen) cudaFreeAsync(otlen, st);
    if (otoff) cudaFreeAsync(otoff, st);
    if (over) cudaFreeAsync(over, st);
    sw16_release(&prep, st);
    sw16_work_release(&work, st);
    sw16_sort_release(&sort, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) rc = -1;
    cudaStreamDestroy(st);
    return rc;
}

/* One SW score pair from host target codes: the wavefront kernel on one warp
 * (int16x2 where no pair can leave 16 bits, else exact int32: no overflow
 * rerun), its descriptors and the codes in one upload to the thread's arena,
 * the output written to the thread's pinned block. */
extern "C" int pb_cuda_sw_single(const pb_device_profile *dp, int open, int gap, const uint8_t *h_codes, int tlen,
                                 pb_pair_out *h_out)
{
    if (pb_cuda_init() != 0) return -1;
    if (!dp->fits8 || !dp->d_prof8 || tlen <= 0 || open + gap > 30000) return -2;
    cudaGetLastError();   /* a launch error below is this call's own */
    const size_t prof_bytes = (size_t)dp->size * dp->lp;
    const bool bias = sw16_bias_ok(dp, open, gap);
    const int rows16 = wave16_rows(&dp, 1);
    const size_t smem16 = wave16_smem(dp, rows16);
    const bool use16 = wave16_ok(dp, tlen, open, gap) && smem16 <= SW16_WAVE_SMEM;
    const size_t smem = use16 ? smem16 : prof_bytes;
    /* the kernels' shared-memory limit raised to this profile (never lowered) */
    {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if ((long long)smem > optin) return -2;
        if (use16) pb_raise_smem((const void *)wave16_kernel(bias, rows16), (int)smem);
        else wave_set_smem((int)smem);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            pb_cuda_set_error("single-pair SW shared memory", cudaGetErrorString(e));
            return -1;
        }
    }
    /* [Sw16Query][toff int64][order, tlen, counter x4: int][out][codes] then the scratch of 8 warps */
    const size_t o_q = 0, o_toff = 32, o_ints = 40, o_out = 64;
    const size_t o_codes = (o_out + sizeof(pb_pair_out) + 15) & ~(size_t)15;
    const size_t up = (o_codes + (size_t)tlen + 16 + 15) & ~(size_t)15;
    const size_t total = up + sizeof(int2) * (size_t)(tlen + 1) * pb::SW16_WARPS;
    char *h = nullptr, *out = nullptr;
    char *d = pb_single_arena(total, up, &h, &out);
    if (!d) { pb_cuda_set_error("single-pair arena", "allocation failed"); return -1; }
    pb::Sw16Query q;
    q.prof8 = dp->d_prof8; q.prof_off = 0; q.qlen = dp->qlen; q.lp = dp->lp; q.posmax = 32767 - dp->mmax - 1;
    memcpy(h + o_q, &q, sizeof q);
    const int ints[6] = {0, tlen, 0, 0, 0, 0};
    memcpy(h + o_ints, ints, sizeof ints);
    memcpy(h + o_codes, h_codes, (size_t)tlen);
    cudaStream_t st = (cudaStream_t)pb_cuda_stream();
    if (cudaMemcpyAsync(d, h, up, cudaMemcpyHostToDevice, st) != cudaSuccess) {
        pb_cuda_set_error("single-pair upload", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    pb::Sw16Params p;
    memset(&p, 0, sizeof p);
    p.open = open; p.gap = gap; p.npairs = 1; p.nq = 1; p.ntasks = 1; p.maxlen = tlen + 1;
    p.nletters = dp->size;
    p.queries = reinterpret_cast<const pb::Sw16Query *>(d + o_q);
    p.prof_all = dp->d_prof8; p.prof_bytes = (int)prof_bytes;
    p.order = reinterpret_cast<const int *>(d + o_ints);
    p.targets = reinterpret_cast<const uint8_t *>(d + o_codes);
    p.toff = reinterpret_cast<const int64_t *>(d + o_toff);
    p.tlen = reinterpret_cast<const int *>(d + o_ints) + 1;
    p.scratch = reinterpret_cast<uint32_t *>(d + up);
    p.out = reinterpret_cast<pb_pair_out *>(out ? out : d + o_out);
    int rl = 8;
    double best = -1.0;
    for (int r = 4; r <= 16; r += 4) {
        const double c = (double)((dp->qlen + 32 * r - 1) / (32 * r)) * (r + 4);
        if (best < 0.0 || c < best) { best = c; rl = r; }
    }
    int *counter = reinterpret_cast<int *>(d + o_ints) + 2;
    if (use16) wave16_kernel(bias, rows16)<<<1, pb::WAVE16_WARPS * 32, smem, st>>>(p, counter);
    else wave_kernel(open >= gap, rl)<<<1, pb::SW16_WARPS * 32, smem, st>>>(p, counter);
    pb_diag_count_launch(1);
    {
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            pb_cuda_set_error("single-pair SW launch", cudaGetErrorString(e));
            return -1;
        }
    }
    if ((!out && cudaMemcpyAsync(h_out, d + o_out, sizeof *h_out, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        pb_cuda_set_error("single-pair SW", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    if (out) memcpy(h_out, out, sizeof *h_out);
    return 0;
}

extern "C" int pb_cuda_align_sw16(const pb_batch *b)
{
    if (b->nprofs != 1 || b->d_prof_index) return pb_cuda_align_exact(b);
    return pb_cuda_align_sw16_multi(b, b->d_out);
}

/* ---- database-search plans: the search as one CUDA graph ------------------ */

namespace {

/* a run's outcome where the host reads it: pairs past 16 bits, error flag */
__global__ void k_plan_status(const int *over, const int *err, volatile int *status)
{
    status[0] = *over;
    status[1] = *err;
}

struct DbPlan {
    cudaStream_t st = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    Sw16Sort sort;
    Sw16Prep prep;
    Sw16Work work;
    bool prepared = false;
    pb_pair_out *o1 = nullptr;
    int *need = nullptr, *counts = nullptr;   /* counts[0..2] lane lists (unused), [4] overflow */
    int *status = nullptr;                    /* pinned: k_plan_status */
    pb_job job;
    pb_batch b;
    std::vector<const pb_device_profile *> profs;
    pb_record *rec = nullptr;
    uint8_t *map = nullptr;                   /* device mapper of plan runs from host memory */
};

void plan_destroy(DbPlan *pl)
{
    if (pl->exec) cudaGraphExecDestroy(pl->exec);
    if (pl->graph) cudaGraphDestroy(pl->graph);
    if (pl->st) {
        if (pl->prepared) sw16_release(&pl->prep, pl->st);
        sw16_work_release(&pl->work, pl->st);
        sw16_sort_release(&pl->sort, pl->st);
        if (pl->o1) cudaFreeAsync(pl->o1, pl->st);
        if (pl->need) cudaFreeAsync(pl->need, pl->st);
        if (pl->counts) cudaFreeAsync(pl->counts, pl->st);
        if (pl->status) cudaFreeHost(pl->status);
        if (pl->map) cudaFreeAsync(pl->map, pl->st);
        cudaStreamSynchronize(pl->st);
        cudaStreamDestroy(pl->st);
    }
    delete pl;
}

}  // namespace

/* A Smith-Waterman score-only database search (every profile of b against
 * every target) whose host-side preparation -- the length order of the
 * targets, the task list, the concatenated profiles, every buffer -- is done
 * once, and whose device work -- the int16x2 score kernel, the count of
 * pairs past the 16-bit range and the width resolution writing d_rec -- is
 * recorded once as a CUDA graph. Running the plan replays the graph on the
 * current contents of b's target buffers (same lengths). Returns -1 when
 * the job is outside what the graph holds (statistics, lane-exact widths,
 * the score kernel's domain). */
extern "C" int pb_cuda_db_plan_create(const pb_job *job, const pb_batch *b, pb_record *d_rec, void **out)
{
    *out = nullptr;
    if (pb_cuda_init() != 0) return -1;
    const int n = b->npairs, nq = b->nprofs;
    const pb_mode *m = &job->mode;
    if (n <= 0 || nq <= 0 || m->alg != PB_SW || m->stats || job->bits < 0) return -1;
    for (int w = 8; w <= 32; w *= 2) if (pb_lane_forced(m, w)) return -1;
    if (b->open + b->gap > 30000 || (long long)n * nq > INT32_MAX) return -1;
    size_t prof_bytes = 0;
    for (int q = 0; q < nq; ++q) {
        const pb_device_profile *dp = b->profs[q];
        if (!dp->fits8 || dp->size != b->profs[0]->size) return -1;
        prof_bytes += (size_t)dp->size * dp->lp;
    }
    if (prof_bytes > SW16_WAVE_SMEM) return -1;
    DbPlan *pl = new DbPlan();
    pl->job = *job;
    pl->profs.assign(b->profs, b->profs + nq);
    pl->b = *b;
    pl->b.profs = pl->profs.data();
    pl->rec = d_rec;
    int rc = 0;
    if (cudaStreamCreateWithFlags(&pl->st, cudaStreamNonBlocking) != cudaSuccess) { pl->st = nullptr; rc = -1; }
    const size_t N = (size_t)n * nq;
    if (rc == 0 && (cudaMallocAsync((void **)&pl->o1, sizeof(pb_pair_out) * N, pl->st) != cudaSuccess ||
                    cudaMallocAsync((void **)&pl->need, sizeof(int) * 3 * (size_t)n, pl->st) != cudaSuccess ||
                    cudaMallocAsync((void **)&pl->counts, sizeof(int) * 8, pl->st) != cudaSuccess ||
                    cudaHostAlloc((void **)&pl->status, sizeof(int) * 2, cudaHostAllocMapped) != cudaSuccess))
        rc = -1;
    if (rc == 0) {
        pb_batch bb = pl->b;
        bb.stats = 0; bb.pad_rows = 0; bb.d_qlim = nullptr; bb.d_tlim = nullptr;
        rc = sw16_sort(&bb, pl->st, &pl->sort);
        if (rc == 0) rc = sw16_prepare(&bb, pl->o1, pl->sort, pl->st, &pl->prep);
        pl->prepared = rc == 0;
        if (rc == 0) rc = sw16_workspace(&pl->prep, pl->st, &pl->work);
    }
    if (rc == 0 && cudaStreamSynchronize(pl->st) != cudaSuccess) rc = -1;
    if (rc == 0 && cudaStreamBeginCapture(pl->st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) rc = -1;
    if (rc == 0) {
        sw16_launch(pl->prep, pl->st);
        cudaMemsetAsync(pl->counts, 0, sizeof(int) * 8, pl->st);
        k_count_overflow<<<148, 256, 0, pl->st>>>(pl->o1, N, pl->counts + 4);
        for (int q = 0; q < nq; ++q)
            pb::launch_resolve_plain(pl->job, pl->o1 + (size_t)q * n, pl->profs[q]->qlen, b->d_tlen, n,
                                     d_rec + (size_t)q * n, pl->need, pl->counts, pl->st);
        k_plan_status<<<1, 1, 0, pl->st>>>(pl->counts + 4, pl->prep.counter + 2, pl->status);
        if (cudaStreamEndCapture(pl->st, &pl->graph) != cudaSuccess) rc = -1;
    }
    if (rc == 0 && cudaGraphInstantiate(&pl->exec, pl->graph, 0) != cudaSuccess) rc = -1;
    if (rc != 0) {
        cudaGetLastError();
        plan_destroy(pl);
        return -1;
    }
    *out = pl;
    return 0;
}

/* Replays the plan's graph; pairs past the 16-bit range (rare: a score
 * above 32767 - max(matrix) - 1) send the whole search once through the
 * batch pipeline, which reruns them in 32 bits. */
extern "C" int pb_cuda_db_plan_run(void *plan)
{
    DbPlan *pl = (DbPlan *)plan;
    if (!pl) return -1;
    if (cudaGraphLaunch(pl->exec, pl->st) != cudaSuccess) return -1;
    pb_diag_count_launch(3 + (long)pl->profs.size());   /* score kernel, overflow count, resolution, status */
    if (cudaStreamSynchronize(pl->st) != cudaSuccess) return -1;
    const int over = pl->status[0], herr = pl->status[1];
    if (herr) {
        fprintf(stderr, "pb_cuda_db_plan_run: a pass wait exceeded its bound\n");
        return -1;
    }
    if (over > 0) return pb_cuda_batch_run(&pl->job, &pl->b, pl->rec);
    return 0;
}

namespace {

__global__ void k_map_inplace(uint8_t *__restrict__ buf, int64_t n, const uint8_t *__restrict__ map)
{
    __shared__ uint8_t smap[256];
    for (int k = threadIdx.x; k < 256; k += blockDim.x) smap[k] = map[k];
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        buf[i] = smap[buf[i]];
}

}  // namespace

/* A plan run from host memory: the targets' characters (the layout the
 * plan was created with) are copied into d_codes and mapped there, the
 * graph replays, and the records come back into h_rec, all on the plan's
 * stream. */
extern "C" int pb_cuda_db_plan_run_host(void *plan, const char *h_chars, size_t nbytes, uint8_t *d_codes,
                                        const uint8_t *mapper256, pb_record *h_rec)
{
    DbPlan *pl = (DbPlan *)plan;
    if (!pl) return -1;
    if (!pl->map) {
        if (cudaMallocAsync((void **)&pl->map, 256, pl->st) != cudaSuccess) return -1;
        if (cudaMemcpyAsync(pl->map, mapper256, 256, cudaMemcpyHostToDevice, pl->st) != cudaSuccess) return -1;
    }
    if (nbytes && cudaMemcpyAsync(d_codes, h_chars, nbytes, cudaMemcpyHostToDevice, pl->st) != cudaSuccess)
        return -1;
    if (nbytes) {
        int dev = 0, nsm = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        const int64_t want = ((int64_t)nbytes + 255) / 256;
        k_map_inplace<<<(int)(want < 2 * nsm ? want : 2 * nsm), 256, 0, pl->st>>>(d_codes, (int64_t)nbytes, pl->map);
        pb_diag_count_launch(1);
    }
    if (pb_cuda_db_plan_run(plan) != 0) return -1;
    const size_t nrec = (size_t)pl->b.npairs * pl->profs.size();
    if (cudaMemcpyAsync(h_rec, pl->rec, sizeof(pb_record) * nrec, cudaMemcpyDeviceToHost, pl->st) != cudaSuccess)
        return -1;
    return cudaStreamSynchronize(pl->st) == cudaSuccess ? 0 : -1;
}

extern "C" void pb_cuda_db_plan_free(void *plan)
{
    if (plan) plan_destroy((DbPlan *)plan);
}
