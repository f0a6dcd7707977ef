// Banded traceback on the GPU: direction bytes, first optimal cell, walk.
//
// k_band_align_warp computes, one job per warp in int32 (lanes across the
// band), the reference's banded_align_scalar (src/algorithm/banded.rs:227-332) — the same direction
// byte org | e_ext << 2 | f_ext << 3 per in-band cell, origin priority
// diagonal > E > F, extension bits only when strictly better — with the early
// exit of the dispatched kernel (rows after the first whose best reaches
// stop_at are not computed, banded_simd.rs:594-596), then follows the
// direction bytes from the first row-major optimal cell back to the start
// exactly as walk (banded.rs:336-403) does and writes the run-length encoded
// operations.  Direction bytes live in a pool in HBM (m x w bytes per job,
// row i at offset i*w, like the reference's dir buffer).  Without the
// direction pool (score-only requests) it returns the score and end cell of
// banded_score (banded.rs:134-224), which traceback_from_end needs.
//
// The widening driver of Engine::traceback / traceback_from_end
// (src/search/engine.rs:1328-1445) runs on the host below: every widening
// round of every unresolved region goes into one launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>
#include <vector>

#include "band_wave.cuh"
#include "saber_gpu.h"

namespace saber {

struct AlignReq {
    const uint8_t* win;  // device window start
    const int16_t* prof; // device query profile (rows c, stride mpad)
    uint64_t dir_off;    // offset of this job's direction bytes in the pool (dir requests)
    uint64_t ops_off;    // offset of this job's op bytes / runs
    int32_t m, n, lo, w; // query length, window length, clipped band, width
    int32_t mpad;
    int32_t stop_at;
    int32_t want_dir;    // 1: direction bytes + walk; 0: score and end cell only
    int32_t zero;        // 0
    const uint32_t* qrow;  // the query's row words (k_align_wave)
};

struct AlignOut {
    int32_t status;  // 1 alignment, 0 none
    int32_t score;
    uint32_t q_start, q_end, s_start, s_end;
    uint32_t n_ops;
    uint32_t run_first;  // first of the n_ops runs, from the job's ops_off
    uint64_t cells;
};

// The walk of one alignment from its best cell (banded.rs:336-403), run by
// one thread over the direction bytes (row stride w), then the run-length
// encoding in forward order.
__device__ void walk_runs(const uint8_t* dir, int64_t w, int64_t lo, int64_t bi, int64_t bk, uint8_t* ob,
                          uint32_t* rr, AlignOut& o) {
    uint32_t nop = 0;
    int state = 0;  // 0 = H, 1 = E (query gap, 'D'), 2 = F (subject gap, 'I')
    int64_t i = bi, k = bk;
    for (;;) {
        const uint8_t d = dir[(size_t)(i * w + k)];
        if (state == 0) {
            const uint8_t org = d & 3;
            if (org == 0) break;
            if (org == 1) {
                ob[nop++] = 'M';
                if (i == 0 || i + lo + k == 0) break;
                i -= 1;
            } else {
                state = org == 2 ? 1 : 2;
            }
        } else if (state == 1) {
            ob[nop++] = 'D';
            const bool ext = (d & 4) != 0;
            k -= 1;
            if (!ext) state = 0;
        } else {
            ob[nop++] = 'I';
            const bool ext = (d & 8) != 0;
            i -= 1;
            k += 1;
            if (!ext) state = 0;
        }
    }
    uint32_t qs = o.q_end, ss = o.s_end, nr = 0;
    for (uint32_t tt = 0; tt < nop; tt++) {
        const uint8_t op = ob[nop - 1 - tt];
        if (op == 'M') {
            qs--;
            ss--;
        } else if (op == 'I') {
            qs--;
        } else {
            ss--;
        }
        if (nr > 0 && (rr[nr - 1] & 0xFFu) == op) rr[nr - 1] += 0x100u;
        else rr[nr++] = 0x100u | op;
    }
    o.q_start = qs;
    o.s_start = ss;
    o.n_ops = nr;
}

// One warp per job: each row's band offsets k = 32c + lane in chunks of 32.
// F and the diagonal come from the previous row (coalesced loads from the
// warp's row buffers); E(i,k) = max over kmin <= j < k of
// H*(i,j) - go - (k-1-j) ge with H* = max(diag + S, F, 0), a warp max-scan of
// H* + j ge -- equal to the scalar recurrence of banded_align_scalar
// (banded.rs:227-332) when go >= ge, because opening a gap from an E-derived
// H never beats extending that E (set_scheme requires go >= ge).  Direction
// bytes, the first row-major best cell, stop_at and the walk are those of
// banded_align_scalar and walk.
__global__ void __launch_bounds__(128) k_band_align_warp(const AlignReq* __restrict__ reqs, uint32_t nreq,
                                                         uint8_t* __restrict__ dir_pool, uint8_t* __restrict__ opbytes,
                                                         uint32_t* __restrict__ runs, int32_t* __restrict__ slabs,
                                                         uint32_t slab_stride, int go, int ge,
                                                         AlignOut* __restrict__ outs) {
    const int NEG = INT32_MIN / 4;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    int32_t* base = slabs + (size_t)warp * slab_stride * 4;
    for (uint32_t t = warp; t < nreq; t += nwarps) {
        const AlignReq rq = reqs[t];
        AlignOut o;
        o.status = 0;
        o.score = 0;
        o.q_start = o.q_end = o.s_start = o.s_end = 0;
        o.n_ops = 0;
        o.run_first = 0;
        o.cells = 0;
        const int64_t m = rq.m, n = rq.n, lo = rq.lo, w = rq.w;
        if (w <= 0) {
            if (lane == 0) outs[t] = o;
            continue;
        }
        int32_t* hp = base;
        int32_t* fp = hp + slab_stride;
        int32_t* hc = fp + slab_stride;
        int32_t* fc = hc + slab_stride;
        for (int64_t k = lane; k <= w; k += 32) hp[k] = fp[k] = hc[k] = fc[k] = NEG;
        __syncwarp();
        uint8_t* dir = rq.want_dir ? dir_pool + rq.dir_off : nullptr;
        int32_t best = 0;
        int64_t bi = 0, bk = 0;
        uint64_t cells = 0;
        const int first_eext = (NEG - ge) > (NEG - go) ? 1 : 0;  // e_ext of a row's first cell
        for (int64_t i = 0; i < m; i++) {
            int64_t kmin = -(i + lo);
            if (kmin < 0) kmin = 0;
            int64_t kmax = n - 1 - i - lo;
            if (kmax > w - 1) kmax = w - 1;
            const int64_t bse = i + lo;
            int tmax = NEG;      // running max of H* + j ge over this row's earlier chunks
            int prevH = NEG, prevE = NEG;  // H and E at k - 1 for lane 0 (carry)
            int rowbest = 0;
            int64_t rowk = 0;
            // only the chunks that hold the row's window cells: the next row
            // reads this row's H and F at its own cells' k and k + 1, inside
            // [kmin - 1, kmax + 1]; at kmin - 1 only as the diagonal of column
            // 0, which is 0 by rule, and entry w stays NEG
            for (int64_t c0 = (kmin / 32) * 32; c0 <= kmax; c0 += 32) {
                const int64_t k = c0 + lane;
                const bool inb = k < w;
                const bool valid = inb && k >= kmin && k <= kmax;
                int f = NEG, hstar = NEG, h1 = 0, fe = 0, fo = 0;
                uint32_t c1 = 0;
                if (valid) {
                    const int64_t j = bse + k;
                    fo = hp[k + 1] - go;
                    fe = fp[k + 1] - ge;
                    f = i >= 1 ? max(fe, fo) : NEG;
                    const int32_t hd = (i >= 1 && j >= 1) ? hp[k] : 0;
                    const int32_t diag = hd + ((int32_t)rq.prof[(size_t)rq.win[j] * rq.mpad + i] - go);
                    c1 = diag > 0;
                    h1 = max(diag, 0);
                    hstar = max(h1, f);
                }
                // E via an exclusive max-scan of H* + k ge (carry from earlier chunks)
                int tv = valid ? hstar + (int)(k * ge) : NEG;
                int incl = tv;
#pragma unroll
                for (int o2 = 1; o2 < 32; o2 <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o2);
                    if (lane >= o2) incl = max(incl, u);
                }
                int excl = __shfl_up_sync(0xffffffffu, incl, 1);
                if (lane == 0) excl = NEG;
                excl = max(excl, tmax);
                int e = NEG;
                if (valid && k > kmin && excl > NEG) e = excl - go - (int)((k - 1) * ge);
                int h = NEG;
                uint8_t d = 0;
                if (valid) {
                    const uint32_t c2 = e > h1;
                    const int32_t h2 = max(h1, e);
                    const uint32_t c3 = f > h2;
                    h = max(h2, f);
                    d = (uint8_t)((c3 ? 3u : (c2 ? 2u : c1)) | ((uint32_t)(fe > fo) << 3));
                }
                // e_ext = E(k-1) - ge > H(k-1) - go (the previous cell of the row)
                int hl = __shfl_up_sync(0xffffffffu, h, 1);
                int el = __shfl_up_sync(0xffffffffu, e, 1);
                if (lane == 0) {
                    hl = prevH;
                    el = prevE;
                }
                if (valid) {
                    const uint32_t eext = k == kmin ? (uint32_t)first_eext : (uint32_t)((el - ge) > (hl - go));
                    d |= (uint8_t)(eext << 2);
                    if (dir) dir[(size_t)(i * w + k)] = d;
                }
                if (inb) {
                    hc[k] = valid ? h : NEG;
                    fc[k] = valid ? f : NEG;
                }
                // the first cell of the row's best
                const int cm = __reduce_max_sync(0xffffffffu, valid ? h : 0);
                if (cm > rowbest) {
                    rowbest = cm;
                    rowk = c0 + (__ffs(__ballot_sync(0xffffffffu, valid && h == cm)) - 1);
                }
                tmax = max(tmax, __shfl_sync(0xffffffffu, incl, 31));
                prevH = __shfl_sync(0xffffffffu, h, 31);
                prevE = __shfl_sync(0xffffffffu, e, 31);
            }
            if (kmin <= kmax) cells += (uint64_t)(kmax - kmin + 1);
            if (rowbest > best) {
                best = rowbest;
                bi = i;
                bk = rowk;
            }
            __syncwarp();
            int32_t* tmp = hp;
            hp = hc;
            hc = tmp;
            tmp = fp;
            fp = fc;
            fc = tmp;
            if (best >= rq.stop_at) break;
        }
        o.cells = cells;
        o.score = best;
        if (best > 0) {
            o.status = 1;
            o.q_end = (uint32_t)(bi + 1);
            o.s_end = (uint32_t)(bi + lo + bk + 1);
        }
        __syncwarp();
        if (lane == 0) {
            if (best > 0 && dir) walk_runs(dir, w, lo, bi, bk, opbytes + rq.ops_off, runs + rq.ops_off, o);
            outs[t] = o;
        }
        __syncwarp();
    }
}

// ---- anti-diagonal sweep (int16 pairs) ----------------------------------------
// The alignment of a band at most kAlignWaveWidth wide: the sweep of
// band_wave.cu, one job on a warp (J x 4 band indices per lane), with the
// direction bits kept per cell and the first step at which each band index
// reached its best.  k_band_align_warp spends a five-shuffle scan per row and
// walks one dependent load at a time; here a row costs two steps of one
// shuffle, and the walk takes the matches of 32 rows at once.  One GB300, a
// whole call by the row kernel -> by this one: 64 queries x 6 M residues (645
// tracebacks) 9.2 -> 6.9 ms, 400 x 150 M bases (3,246 kilobase tracebacks)
// 59.3 -> 36.9 ms, 11,000 x 150 M residues (108 k) 600 -> 574 ms.
//
// Directions: one byte per cell, bit 0 diagonal > 0, 1 E > max(diagonal, 0),
// 2 F above both (the origin priority diagonal > E > F), 3 and 4: the E and F
// leaving this cell extend (strictly better than opening here).  A word holds
// the four band indices of a lane and J; pair of steps `it` of a job is a row
// of ceil(w / 4) words, so a warp's stores are contiguous.
//
// The reference stops after the first row whose best reaches stop_at.  The
// sweep goes on for the rest of the rows above the first cell that reached it
// and takes the first row-major cell of the best score: the same cell when
// that score is stop_at itself.  When it is higher (or outside int16) the job
// is flagged kAlignRedo and runs through k_band_align_warp.
constexpr int kAlignRedo = 3;

template <int J>
__device__ __forceinline__ void align_wave(const AlignReq& rq, uint32_t* __restrict__ dir, uint32_t* __restrict__ rr,
                                           int lane, const uint8_t* tab, int go, int ge, AlignOut& o) {
    const int m = rq.m, n = rq.n, lo = rq.lo, w = rq.w;
    int s0, nit;
    wv_span(m, n, lo, w, s0, nit);
    const uint32_t ngo2 = wv_pk2(-go), nge2 = wv_pk2(-ge), neg2 = wv_pk2(kNeg16);
    const uint32_t* qrow = rq.qrow;
    const uint8_t* win = rq.win;
    int i0 = s0 / 2 - 2 * J * lane;
    int c0 = s0 / 2 + 2 * J * lane + lo;
    const int istart = i0;
    const uint32_t pitch = (uint32_t)(w + 3) / 4;
    const bool stores = J * lane * 4 < w;
    const int words = min(J, (int)pitch - J * lane);  // of this lane, when it stores

    uint32_t Ge[J], Go[J], E[J], F[J], keep_e[J], keep_o[J], R[2 * J], C[2 * J + 1], B[J];
    uint32_t best_e[J], best_o[J];
    int at_e[2 * J], at_o[2 * J];
#pragma unroll
    for (int j = 0; j < J; j++) {
        Ge[j] = Go[j] = ngo2;
        E[j] = F[j] = neg2;
        best_e[j] = best_o[j] = 0;
        at_e[2 * j] = at_e[2 * j + 1] = at_o[2 * j] = at_o[2 * j + 1] = 0;
        const int k = 4 * J * lane + 4 * j;
        keep_e[j] = (k < w ? 0xFFFFu : 0u) | (k + 2 < w ? 0xFFFF0000u : 0u);
        keep_o[j] = (k + 1 < w ? 0xFFFFu : 0u) | (k + 3 < w ? 0xFFFF0000u : 0u);
        const uint32_t ra = wv_row(qrow, i0 - 2 * j, m), rb = wv_row(qrow, i0 - 2 * j - 1, m);
        R[2 * j] = ra & 0xFFFFu;
        R[2 * j + 1] = rb & 0xFFFFu;
        B[j] = wv_prmt(ra, rb, 0x7632);
    }
#pragma unroll
    for (int r = 0; r <= 2 * J; r++) C[r] = 2 * wv_col(win, c0 + r, n);
    uint32_t qn[kWaveAhead], sn[kWaveAhead];
#pragma unroll
    for (int t = 0; t < kWaveAhead; t++) {
        qn[t] = wv_row(qrow, i0 + 1 + t, m);
        sn[t] = wv_col(win, c0 + 2 * J + 1 + t, n);
    }
    i0 += kWaveAhead;
    c0 += 2 * J + kWaveAhead;
    // zero, loaded: with an immediate 0 the packed maximum of nvcc 13.0 returns
    // wrong predicates (checked against all the other operand kinds)
    const uint32_t zero2 = (uint32_t)rq.zero;
    const int stop = min(rq.stop_at, 32767);
    int iend = nit;
    bool found = false;
    // one cell pair: H and the bits of both cells (their bytes at bit b and b + 16)
    auto cells = [&](uint32_t diag, uint32_t Ein, uint32_t Fin, uint32_t keep, uint32_t& G, uint32_t& Eo, uint32_t& Fo,
                     uint32_t& best, int& at_lo, int& at_hi, int it, uint32_t& word, int b) {
        bool ph, pl;
        const uint32_t h1 = __vibmax_s16x2(zero2, diag, &ph, &pl);
        if (!pl) word |= 1u << b;
        if (!ph) word |= 1u << (b + 16);
        const uint32_t h2 = __vibmax_s16x2(h1, Ein, &ph, &pl);
        if (!pl) word |= 2u << b;
        if (!ph) word |= 2u << (b + 16);
        const uint32_t h3 = __vibmax_s16x2(h2, Fin, &ph, &pl);
        if (!pl) word |= 4u << b;
        if (!ph) word |= 4u << (b + 16);
        const uint32_t H = h3 & keep;
        G = __vadd2(H, ngo2);
        Eo = __vibmax_s16x2(G, __vadd2(Ein, nge2), &ph, &pl);
        if (!pl) word |= 8u << b;
        if (!ph) word |= 8u << (b + 16);
        Fo = __vibmax_s16x2(G, __vadd2(Fin, nge2), &ph, &pl);
        if (!pl) word |= 16u << b;
        if (!ph) word |= 16u << (b + 16);
        best = __vibmax_s16x2(best, H, &ph, &pl);
        at_lo = pl ? at_lo : it;
        at_hi = ph ? at_hi : it;
    };
    for (int it0 = 0; it0 < iend; it0 += kWaveAhead) {
#pragma unroll
        for (int t = 0; t < kWaveAhead; t++) {
            const int it = it0 + t;
            uint32_t word[J];
#pragma unroll
            for (int j = 0; j < J; j++) word[j] = 0;
            uint32_t left = __shfl_up_sync(0xffffffffu, E[J - 1], 1);
            if (lane == 0) left = neg2;
#pragma unroll
            for (int j = 0; j < J; j++) {
                const uint32_t own = E[j];
                const uint32_t Ein = wv_prmt(left, own, 0x5432);
                left = own;
                const uint32_t Fin = F[j];
                const uint32_t ds = __vadd2(Ge[j], wv_sub(tab, R[2 * j], C[2 * j], R[2 * j + 1], C[2 * j + 1], B[j]));
                cells(ds, Ein, Fin, keep_e[j], Ge[j], E[j], F[j], best_e[j], at_e[2 * j], at_e[2 * j + 1], it, word[j], 0);
            }
            uint32_t down = __shfl_down_sync(0xffffffffu, F[0], 1);
            if (lane == 31) down = neg2;
#pragma unroll
            for (int j = 0; j < J; j++) {
                const uint32_t Ein = E[j];
                const uint32_t Fin = wv_prmt(F[j], j + 1 < J ? F[j + 1 < J ? j + 1 : j] : down, 0x5432);
                const uint32_t ds =
                    __vadd2(Go[j], wv_sub(tab, R[2 * j], C[2 * j + 1], R[2 * j + 1], C[2 * j + 2], B[j]));
                cells(ds, Ein, Fin, keep_o[j], Go[j], E[j], F[j], best_o[j], at_o[2 * j], at_o[2 * j + 1], it, word[j], 8);
            }
            if (stores && it < nit) {
                uint32_t* d = dir + (size_t)it * pitch + J * lane;
#pragma unroll
                for (int j = 0; j < J; j++)
                    if (j < words) d[j] = word[j];
            }
#pragma unroll
            for (int j = J - 1; j > 0; j--) B[j] = wv_prmt(B[j - 1], B[j], 0x5432);
            B[0] = wv_prmt(qn[t], B[0], 0x5432);
#pragma unroll
            for (int r = 2 * J - 1; r > 0; r--) R[r] = R[r - 1];
            R[0] = qn[t] & 0xFFFFu;
#pragma unroll
            for (int r = 0; r < 2 * J; r++) C[r] = C[r + 1];
            C[2 * J] = 2 * sn[t];
            i0++;
            c0++;
            qn[t] = wv_row(qrow, i0, m);
            sn[t] = wv_col(win, c0, n);
        }
        if (!found) {
            uint32_t b = 0;
#pragma unroll
            for (int j = 0; j < J; j++) b = __vimax3_s16x2(b, best_e[j], best_o[j]);
            const bool hit = (int)(b & 0xFFFFu) >= stop || (int)(b >> 16) >= stop;
            if (__any_sync(0xffffffffu, hit)) {
                // every row up to the one that reached it is complete w
                // anti-diagonals after the last one swept
                found = true;
                iend = min(iend, it0 + kWaveAhead + (w + 1) / 2);
            }
        }
    }
    // the first row-major cell of the best score
    int bs = 0, bi = INT_MAX, bk = INT_MAX;
    auto take = [&](uint32_t v, int it, int j, int half, int par) {
        const int sc = half ? (int)(v >> 16) : (int)(v & 0xFFFFu);
        const int i = istart + it - 2 * j - half, k = 4 * J * lane + 4 * j + par + 2 * half;
        if (sc > bs || (sc == bs && (i < bi || (i == bi && k < bk)))) {
            bs = sc;
            bi = i;
            bk = k;
        }
    };
#pragma unroll
    for (int j = 0; j < J; j++) {
        take(best_e[j], at_e[2 * j], j, 0, 0);
        take(best_o[j], at_o[2 * j], j, 0, 1);
        take(best_e[j], at_e[2 * j + 1], j, 1, 0);
        take(best_o[j], at_o[2 * j + 1], j, 1, 1);
    }
    const int best = __reduce_max_sync(0xffffffffu, bs);
    bi = __reduce_min_sync(0xffffffffu, bs == best ? bi : INT_MAX);
    {
        // k of the lanes that hold row bi at the best score
        int kk = INT_MAX;
        auto at_row = [&](uint32_t v, int it, int j, int half, int par) {
            const int sc = half ? (int)(v >> 16) : (int)(v & 0xFFFFu);
            if (sc == best && istart + it - 2 * j - half == bi) kk = min(kk, 4 * J * lane + 4 * j + par + 2 * half);
        };
#pragma unroll
        for (int j = 0; j < J; j++) {
            at_row(best_e[j], at_e[2 * j], j, 0, 0);
            at_row(best_o[j], at_o[2 * j], j, 0, 1);
            at_row(best_e[j], at_e[2 * j + 1], j, 1, 0);
            at_row(best_o[j], at_o[2 * j + 1], j, 1, 1);
        }
        bk = __reduce_min_sync(0xffffffffu, kk);
    }
    o.score = best;
    if (best >= kLimit16 || best > rq.stop_at) {
        o.status = kAlignRedo;
        return;
    }
    // rows the reference computes: up to the one that reached stop_at
    {
        const int64_t mm = best >= rq.stop_at ? bi + 1 : m;
        int64_t l = lo, h = (int64_t)lo + w - 1;
        o.cells = clip_band(mm, n, l, h) > 0 ? band_cells(mm, n, l, h) : 0;
    }
    if (best <= 0) return;
    o.status = 1;
    o.q_end = (uint32_t)(bi + 1);
    o.s_end = (uint32_t)(bi + lo + bk + 1);

    // The walk (banded.rs:336-403), every lane in the same state: lane t holds
    // the direction word of pair of steps top - t in the current column of four
    // band indices, so a run of matches (the band index stays, the pair of steps
    // goes down by one) is a ballot.  Runs are written backwards from the end
    // of the job's area.
    __syncwarp();
    const uint32_t cap = (uint32_t)m + (uint32_t)n + 2u;
    uint32_t nr = 0, op = 0, len = 0, qs = o.q_end, ss = o.s_end;
    auto emit = [&](uint32_t c, uint32_t l) {
        if (c == op) {
            len += l;
            return;
        }
        if (len && lane == 0) rr[cap - 1 - nr] = (len << 8) | op;
        nr += len != 0;
        op = c;
        len = l;
    };
    int i = bi, k = bk, state = 0, top = -1, col = -1;
    uint32_t mine = 0;
    for (uint32_t guard = 0; guard < 2 * cap; guard++) {
        const int it = (2 * i + k - s0) >> 1;
        if (i < 0 || k < 0 || k >= w || it < 0 || it >= nit) break;  // (outside the sweep: never reached)
        if (col != (k >> 2) || top - it >= 32) {
            col = k >> 2;
            top = it;
            mine = it - lane >= 0 ? dir[(size_t)(it - lane) * pitch + col] : 0u;
        }
        const uint32_t byte = (mine >> (8 * (k & 3))) & 0xFFu;
        const int off = top - it;
        const uint32_t d = __shfl_sync(0xffffffffu, byte, off);
        // arriving from a gap: does it go on here?
        if (state == 1 && !(d & 8u)) state = 0;
        else if (state == 2 && !(d & 16u)) state = 0;
        if (state == 0) {
            if (!(d & 7u)) break;  // H = 0
            if ((d & 6u) == 0) {
                const uint32_t run = __ballot_sync(0xffffffffu, (byte & 7u) == 1u) >> off;
                const int j = i + lo + k;
                int l = run == 0xFFFFFFFFu ? 32 : __ffs(~run) - 1;
                const int lim = min(i, j) + 1;
                const bool end = l >= lim;
                if (end) l = lim;
                emit('M', (uint32_t)l);
                qs -= l;
                ss -= l;
                if (end) break;
                i -= l;
                continue;
            }
            state = (d & 4u) ? 2 : 1;
        }
        if (state == 1) {
            emit('D', 1u);
            ss--;
            k -= 1;
        } else {
            emit('I', 1u);
            qs--;
            i -= 1;
            k += 1;
        }
    }
    emit(0u, 0u);
    o.q_start = qs;
    o.s_start = ss;
    o.n_ops = nr;
    o.run_first = cap - nr;
}

__global__ void __launch_bounds__(128, 4) k_align_wave(const AlignReq* __restrict__ reqs, uint32_t nreq,
                                                       uint8_t* dir_pool, uint32_t* __restrict__ runs,
                                                       const int32_t* __restrict__ matrix, int go, int ge,
                                                       uint32_t* __restrict__ next, AlignOut* __restrict__ outs) {
    __shared__ __align__(4) int16_t tab[25 * kWaveRow / 2];
    wv_table(tab, matrix, go);
    __syncthreads();
    const uint8_t* tb = reinterpret_cast<const uint8_t*>(tab);
    const int lane = threadIdx.x & 31;
    for (;;) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(next, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= nreq) break;
        const AlignReq rq = reqs[t];
        AlignOut o;
        o.status = 0;
        o.score = 0;
        o.q_start = o.q_end = o.s_start = o.s_end = 0;
        o.n_ops = 0;
        o.run_first = 0;
        o.cells = 0;
        uint32_t* dir = reinterpret_cast<uint32_t*>(dir_pool + rq.dir_off);
        uint32_t* rr = runs + rq.ops_off;
        if (rq.w > 256) align_wave<4>(rq, dir, rr, lane, tb, go, ge, o);
        else if (rq.w > 128) align_wave<2>(rq, dir, rr, lane, tb, go, ge, o);
        else align_wave<1>(rq, dir, rr, lane, tb, go, ge, o);
        if (lane == 0) outs[t] = o;
        __syncwarp();
    }
}

cudaError_t launch_align_wave(unsigned sm_count, cudaStream_t s, const AlignReq* reqs, uint32_t nreq, uint8_t* dir_pool,
                              uint32_t* runs, const int32_t* matrix, int go, int ge, uint32_t* next, AlignOut* outs) {
    const unsigned grid = std::min<unsigned>(sm_count * 4, (nreq + 3) / 4);
    k_align_wave<<<grid, 128, 0, s>>>(reqs, nreq, dir_pool, runs, matrix, go, ge, next, outs);
    return cudaGetLastError();
}

cudaError_t launch_band_align(unsigned grid, cudaStream_t s, const AlignReq* reqs, uint32_t nreq, uint8_t* dir_pool,
                              uint8_t* opbytes, uint32_t* runs, int32_t* slabs, uint32_t slab_stride, int go, int ge,
                              AlignOut* outs) {
    // (set_scheme guarantees go >= ge, the condition of the warp kernel's E scan)
    k_band_align_warp<<<grid, 128, 0, s>>>(reqs, nreq, dir_pool, opbytes, runs, slabs, slab_stride, go, ge, outs);
    return cudaGetLastError();
}

}  // namespace saber
