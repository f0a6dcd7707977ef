// Banded affine-gap Smith-Waterman, one job on 8, 9, 16 or 32 lanes, or on a
// block's 128 (int16 pairs): the jobs whose sweep in one lane of k_band_fast
// would outlast the rest of the batch, and narrow bands.  Semantics as in
// band_kernels.cu.
//
// The band is swept along anti-diagonals s = 2 i + k of its (row i, band
// index k = j - i - lo) coordinates.  A lane holds 4 J consecutive band
// indices k0 = 4 J l ..: the even ones in J registers of pairs (k, k + 2),
// the odd ones in J more.  The cells of one anti-diagonal have the parity of
// s, so an even step updates the even registers from the odd ones and the
// other way round:
//   left neighbour (i, k - 1)    at s - 1, the other parity
//   upper neighbour (i - 1, k + 1) at s - 1, the other parity
//   diagonal (i - 1, k)          at s - 2, the same register
// so every lane works on every step whatever the band's width, one warp
// shuffle per step crosses lanes, and nothing goes through memory.  A job
// takes 2 rows + w steps, against (strips x (w + 15)) steps of 16 dependent
// rows in one lane of the strip kernel.
//
// A lane's rows at one step are i0, i0 - 1, ..., i0 - 2J + 1 and its columns
// c0 .. c0 + 2J; both windows advance by one per two steps, so one query
// letter and one subject letter enter per lane and two steps (fetched four
// pairs of steps ahead).  A row meets column c in an even step and column
// c + 1 in the odd step after it, so the scores (S + go) are kept in shared
// memory per code and pair of column codes, two bytes each: one 16-bit read
// serves both steps, and a byte permute widens it (31 KB; schemes whose scores
// do not fit in a byte read a 25 x 25 int16 table per step).  The packed query
// bias of the row pair is added.
//
// Bound: the ALU pipe (75 % busy at 100 k jobs; L1 80 %, issue slots 70 %).
// With the int16 table alone it was L1 wavefronts of the gathers (95 %): 100 k
// jobs 1.69 -> 1.41 ms, 300 k 4.77 -> 3.91, 1 M 15.5 -> 12.7, against 8.2 in
// the strip kernel, whose rate needs a full device; this one reaches
// 1.6e12 cells/s from a few thousand jobs on.
// One GB300: 3,001 host jobs (half-widths 4..64) 1.78 -> 0.26 ms a call, 40
// full windows of a 310-residue query 0.86 -> 0.26 ms, 2 x 3,662 kilobase DNA
// bands 16.5 -> 4 ms of scoring.
//
// Cells left of column 0 or above row 0 hold H = 0 and E, F <= 0 from the
// initial state on (their score is the sentinel), which is what the
// recurrence reads there; cells past the last row or column hold values below
// the optimum and feed no cell of the window; cells past the band (k >= w in
// the last lanes) are held at H = 0 by a mask, so that neither E nor F carries
// a score across the band's edge.
#include "band_wave.cuh"

namespace saber {

constexpr unsigned kWaveThreads = 128;

// Byte permute with sign replication (a selector nibble 8 | b: the sign of byte b).
__device__ __forceinline__ uint32_t wv_sext(uint32_t x, uint32_t y, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(y), "r"(sel));
    return d;
}

// Jobs [task * 32 / L, ...) of one (L, J) class of the sorted list, one per
// group of L lanes.  L = 128: one job on the block's four warps, whose edge
// lanes pass E and F through shared memory (xch), a barrier per step.
template <int L, int J, bool P8>
__device__ __forceinline__ void wave_task(const WaveArgs& a, const uint32_t* __restrict__ list, uint32_t njobs,
                                          uint32_t task, int lane, const uint8_t* tab, uint32_t* xch) {
    constexpr bool kBlock = L > 32;
    constexpr int G = kBlock ? 1 : 32 / L;
    const int gl = kBlock ? (int)threadIdx.x : lane % L, wib = (int)threadIdx.x >> 5;
    const uint32_t pos = kBlock ? task : task * G + (uint32_t)(lane / L);
    const bool has = pos < njobs && (kBlock || lane < G * L);
    uint32_t jid = 0;
    int m = 0, n = 0, lo = 0, w = 0, s0 = 0, nit = 0;
    const uint32_t* qrow = a.qrow;
    const uint8_t* win = a.res;
    if (has) {
        jid = list[pos];
        const saber_band_job jj = a.jobs[jid];
        const uint64_t q0 = a.qoffs[jj.query];
        const int64_t mm = (int64_t)(a.qoffs[jj.query + 1] - q0);
        int64_t l64 = jj.band_lo, h64 = jj.band_hi;
        w = (int)clip_band(mm, jj.win_len, l64, h64);
        m = (int)mm;
        n = (int)jj.win_len;
        lo = (int)l64;
        qrow += q0;
        win += jj.win_begin;
        wv_span(m, n, lo, w, s0, nit);
    }
    const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)nit);
    const int go = a.go;
    const uint32_t ngo2 = wv_pk2(-go), nge2 = wv_pk2(-a.ge), neg2 = wv_pk2(kNeg16);
    int i0 = s0 / 2 - 2 * J * gl;
    int c0 = s0 / 2 + 2 * J * gl + lo;

    // C: columns 0 .. 2J as offsets (int16 table), or column pairs 0 .. 2J - 1
    // (pair table; `last` is the code of column 2J)
    uint32_t Ge[J], Go[J], E[J], F[J], keep_e[J], keep_o[J], R[2 * J], C[2 * J + 1], B[J], last = 0;
#pragma unroll
    for (int j = 0; j < J; j++) {
        Ge[j] = Go[j] = ngo2;
        E[j] = F[j] = neg2;
        const int k = 4 * J * gl + 4 * j;
        keep_e[j] = (k < w ? 0xFFFFu : 0u) | (k + 2 < w ? 0xFFFF0000u : 0u);
        keep_o[j] = (k + 1 < w ? 0xFFFFu : 0u) | (k + 3 < w ? 0xFFFF0000u : 0u);
        const uint32_t ra = wv_row(qrow, i0 - 2 * j, m), rb = wv_row(qrow, i0 - 2 * j - 1, m);
        R[2 * j] = ra & 0xFFFFu;
        R[2 * j + 1] = rb & 0xFFFFu;
        B[j] = wv_prmt(ra, rb, 0x7632);
    }
#pragma unroll
    for (int r = 0; r <= 2 * J; r++) C[r] = wv_col(win, c0 + r, n);
    if (P8) {
        last = C[2 * J];
#pragma unroll
        for (int r = 0; r < 2 * J; r++) C[r] = 50 * C[r] + 2 * C[r + 1];
    } else {
#pragma unroll
        for (int r = 0; r <= 2 * J; r++) C[r] *= 2;
    }
    // letters of the next kWaveAhead pairs of steps
    uint32_t qn[kWaveAhead], sn[kWaveAhead];
#pragma unroll
    for (int t = 0; t < kWaveAhead; t++) {
        qn[t] = wv_row(qrow, i0 + 1 + t, m);
        sn[t] = wv_col(win, c0 + 2 * J + 1 + t, n);
    }
    i0 += kWaveAhead;
    c0 += 2 * J + kWaveAhead;
    uint32_t best = 0;
    if (kBlock) {
        if (lane == 31) xch[wib] = neg2;
        __syncthreads();
    }
    for (int it = 0; it < nmax; it += kWaveAhead) {
#pragma unroll
        for (int t = 0; t < kWaveAhead; t++) {
            uint32_t X[P8 ? J : 1], Y[P8 ? J : 1];  // both steps' scores of the rows 2j and 2j + 1
            if (P8) {
#pragma unroll
                for (int j = 0; j < J; j++) {
                    X[P8 ? j : 0] = *reinterpret_cast<const uint16_t*>(tab + R[2 * j] + C[2 * j]);
                    Y[P8 ? j : 0] = *reinterpret_cast<const uint16_t*>(tab + R[2 * j + 1] + C[2 * j + 1]);
                }
            }
            // even step: E, F come in from the odd band indices
            uint32_t left = __shfl_up_sync(0xffffffffu, E[J - 1], 1);
            if (kBlock && lane == 0 && wib > 0) left = xch[wib - 1];
            if (gl == 0) left = neg2;
#pragma unroll
            for (int j = 0; j < J; j++) {
                const uint32_t own = E[j];
                const uint32_t Ein = wv_prmt(left, own, 0x5432);
                left = own;
                const uint32_t Fin = F[j];
                const uint32_t ds =
                    __vadd2(Ge[j], P8 ? __vadd2(wv_sext(X[P8 ? j : 0], Y[P8 ? j : 0], 0xC480u), B[j])
                                      : wv_sub(tab, R[2 * j], C[2 * j], R[2 * j + 1], C[2 * j + 1], B[j]));
                const uint32_t H = __vimax3_s16x2_relu(Ein, Fin, ds) & keep_e[j];
                const uint32_t Gv = __vadd2(H, ngo2);
                Ge[j] = Gv;
                E[j] = __viaddmax_s16x2(Ein, nge2, Gv);
                F[j] = __viaddmax_s16x2(Fin, nge2, Gv);
                best = __vmaxs2(best, H);
            }
            if (kBlock) {
                if (lane == 0) xch[4 + wib] = F[0];
                __syncthreads();
            }
            // odd step: from the even ones
            uint32_t down = __shfl_down_sync(0xffffffffu, F[0], 1);
            if (kBlock && lane == 31 && gl != L - 1) down = xch[5 + wib];
            if (gl == L - 1) down = neg2;
#pragma unroll
            for (int j = 0; j < J; j++) {
                const uint32_t Ein = E[j];
                const uint32_t Fin = wv_prmt(F[j], j + 1 < J ? F[j + 1 < J ? j + 1 : j] : down, 0x5432);
                const uint32_t ds =
                    __vadd2(Go[j], P8 ? __vadd2(wv_sext(X[P8 ? j : 0], Y[P8 ? j : 0], 0xD591u), B[j])
                                      : wv_sub(tab, R[2 * j], C[2 * j + 1], R[2 * j + 1], C[2 * j + 2], B[j]));
                const uint32_t H = __vimax3_s16x2_relu(Ein, Fin, ds) & keep_o[j];
                const uint32_t Gv = __vadd2(H, ngo2);
                Go[j] = Gv;
                E[j] = __viaddmax_s16x2(Ein, nge2, Gv);
                F[j] = __viaddmax_s16x2(Fin, nge2, Gv);
                best = __vmaxs2(best, H);
            }
            if (kBlock) {
                if (lane == 31) xch[wib] = E[J - 1];
                __syncthreads();
            }
            // the windows advance by one row and one column
#pragma unroll
            for (int j = J - 1; j > 0; j--) B[j] = wv_prmt(B[j - 1], B[j], 0x5432);
            B[0] = wv_prmt(qn[t], B[0], 0x5432);
#pragma unroll
            for (int r = 2 * J - 1; r > 0; r--) R[r] = R[r - 1];
            R[0] = qn[t] & 0xFFFFu;
            if (P8) {
#pragma unroll
                for (int r = 0; r < 2 * J - 1; r++) C[r] = C[r + 1];
                C[2 * J - 1] = 50 * last + 2 * sn[t];
                last = sn[t];
            } else {
#pragma unroll
                for (int r = 0; r < 2 * J; r++) C[r] = C[r + 1];
                C[2 * J] = 2 * sn[t];
            }
            i0++;
            c0++;
            qn[t] = wv_row(qrow, i0, m);
            sn[t] = wv_col(win, c0, n);
        }
    }
    int sc = max((int)(best & 0xFFFFu), (int)(best >> 16));  // H >= 0
    // the group's maximum in its first lane (lanes past the group's end add
    // nothing: their values are masked out)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int v = __shfl_down_sync(0xffffffffu, sc, o);
        if (o < L && gl + o < L) sc = max(sc, v);
    }
    if (kBlock) {
        __syncthreads();  // (xch may still be read)
        if (lane == 0) xch[wib] = (uint32_t)sc;
        __syncthreads();
        sc = (int)max(max(xch[0], xch[1]), max(xch[2], xch[3]));
        __syncthreads();
    }
    if (has && gl == 0) {
        if (sc >= kLimit16) a.rescue[atomicAdd(a.rescue_count, 1u)] = jid;
        else a.scores[jid] = sc;
    }
}

// Persistent warps over warp tasks of the classes, widest bands first; within
// a class the list is largest first.
template <bool P8>
__global__ void __launch_bounds__(kWaveThreads, 4) k_band_wave(WaveArgs a) {
    __shared__ __align__(16) uint8_t tab[(kWavePairBytes + 15) / 16 * 16];
    __shared__ uint32_t xch[8];
    if (P8) {
        // every load of the copy in flight at once: a batch of a few jobs waits for it
        constexpr int kVec = (kWavePairBytes + 15) / 16, kPer = (kVec + kWaveThreads - 1) / kWaveThreads;
        uint4 v[kPer];
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            const int t = i * kWaveThreads + threadIdx.x;
            if (t < kVec) v[i] = __ldg(reinterpret_cast<const uint4*>(a.pairs) + t);
        }
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            const int t = i * kWaveThreads + threadIdx.x;
            if (t < kVec) reinterpret_cast<uint4*>(tab)[t] = v[i];
        }
    } else {
        wv_table(reinterpret_cast<int16_t*>(tab), a.matrix, a.go);
    }
    __syncthreads();
    const uint8_t* tb = tab;
    const int lane = threadIdx.x & 31;
    uint32_t n[kWaveClasses], tasks[kWaveClasses], total = 0;
#pragma unroll
    for (int c = 0; c < kWaveClasses; c++) {
        n[c] = a.counts[c];
        const uint32_t per = c < 4 ? 1u : c - 2u;  // jobs per warp
        tasks[c] = (n[c] + per - 1) / per;
        total += tasks[c];
    }
    const uint32_t* list = a.order + (a.skip0 ? *a.skip0 : 0u) + (a.skip1 ? *a.skip1 : 0u);
    // Few wide bands: one on a whole block (8 or 4 band indices a lane) instead
    // of 32 or 16 a lane on one warp.  The longest job is then the launch: 40
    // full windows of a 310-residue query 383 -> 257 us a call.  Many of them
    // keep every warp busy by themselves, and a lane's sets share its overheads.
    if (n[0] + n[1] <= 2 * gridDim.x) {
        for (uint32_t p = blockIdx.x; p < n[0] + n[1]; p += gridDim.x) {
            if (p < n[0]) wave_task<128, 2, P8>(a, list, n[0], p, lane, tb, xch);
            else wave_task<128, 1, P8>(a, list + n[0], n[1], p - n[0], lane, tb, xch);
        }
        total -= tasks[0] + tasks[1];
        tasks[0] = tasks[1] = 0;
    }
    for (;;) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(a.task_counter, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= total) break;
        const uint32_t* l = list;
        if (t < tasks[0]) {
            wave_task<32, 8, P8>(a, l, n[0], t, lane, tb, xch);
            continue;
        }
        t -= tasks[0];
        l += n[0];
        if (t < tasks[1]) {
            wave_task<32, 4, P8>(a, l, n[1], t, lane, tb, xch);
            continue;
        }
        t -= tasks[1];
        l += n[1];
        if (t < tasks[2]) {
            wave_task<32, 2, P8>(a, l, n[2], t, lane, tb, xch);
            continue;
        }
        t -= tasks[2];
        l += n[2];
        if (t < tasks[3]) {
            wave_task<32, 1, P8>(a, l, n[3], t, lane, tb, xch);
            continue;
        }
        t -= tasks[3];
        l += n[3];
        if (t < tasks[4]) {
            wave_task<16, 1, P8>(a, l, n[4], t, lane, tb, xch);
            continue;
        }
        t -= tasks[4];
        l += n[4];
        if (t < tasks[5]) {
            wave_task<9, 1, P8>(a, l, n[5], t, lane, tb, xch);
            continue;
        }
        t -= tasks[5];
        l += n[5];
        wave_task<8, 1, P8>(a, l, n[6], t, lane, tb, xch);
    }
}

// Pair table of a scheme (kWavePairBytes, 16-byte aligned).
__global__ void k_wave_pairs(const int32_t* __restrict__ matrix, int go, uint8_t* __restrict__ pairs) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < kWavePairBytes / 2; t += gridDim.x * blockDim.x) {
        const int q = t / 625, c = t / 25 % 25, d = t % 25;
        const int x = q < 24 && c < 24 ? matrix[q * 24 + c] + go : -128, y = q < 24 && d < 24 ? matrix[q * 24 + d] + go : -128;
        pairs[2 * t] = (uint8_t)(int8_t)x;
        pairs[2 * t + 1] = (uint8_t)(int8_t)y;
    }
}
cudaError_t launch_wave_pairs(cudaStream_t s, const int32_t* matrix, int go, uint8_t* pairs) {
    k_wave_pairs<<<31, 256, 0, s>>>(matrix, go, pairs);
    return cudaGetLastError();
}

cudaError_t launch_band_wave(unsigned sm_count, cudaStream_t s, const WaveArgs& a) {
    if (a.pairs) k_band_wave<true><<<sm_count * 4, kWaveThreads, 0, s>>>(a);
    else k_band_wave<false><<<sm_count * 4, kWaveThreads, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace saber
