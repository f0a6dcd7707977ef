// Learned triage of candidate regions: a 3-layer MLP (24 features -> 256 ->
// 256 -> 1 logit, ReLU) with bf16 weights and fp32 accumulation, trained on
// the GPU by the kernels below (forward, backward, Adam) on labels that the
// plain search produces (the region yields a reported hit at the E-value
// cut), and used by the batch engine to drop candidate regions before the
// banded scoring.  Every surviving region is still scored exactly; the plain
// path (no model installed) is unchanged.  No reference counterpart: the
// reference scores every candidate region.
//
// Model layout (floats, host and ABI): W1[32][256] (input-major, rows 24..31
// unused), b1[256], W2[256][256], b2[256], W3[256], b3, mu[32], isd[32]
// (the input normalisation x' = (x - mu) * isd).  The forward pass rounds the
// weights to bf16; training keeps fp32 master weights.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "runtime.cuh"

namespace saber {

static_assert(SABER_TRIAGE_ROW_FLOATS == 32, "feature row width");
constexpr int kTIn = 32, kTFeat = 24, kTHid = 256;
constexpr size_t kOffW1 = 0, kOffB1 = kOffW1 + kTIn * kTHid, kOffW2 = kOffB1 + kTHid,
                 kOffB2 = kOffW2 + kTHid * kTHid, kOffW3 = kOffB2 + kTHid, kOffB3 = kOffW3 + kTHid,
                 kOffMu = kOffB3 + 1, kOffIsd = kOffMu + kTIn, kModelFloats = kOffIsd + kTIn;
static_assert(kModelFloats == SABER_TRIAGE_MODEL_FLOATS, "model layout");

// ---- per-sequence composition features --------------------------------------
// One warp per sequence: Shannon entropy of the 20 standard residues (bits),
// the fraction of positions starting a 12-residue window with at most 4
// distinct residues (low complexity), the largest residue frequency, and the
// fraction of non-standard codes.
__global__ void k_seq_feats(const uint8_t* __restrict__ codes, const uint64_t* __restrict__ offs, uint64_t n,
                            float4* __restrict__ out) {
    __shared__ uint32_t hist[8][24];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint64_t s = (uint64_t)blockIdx.x * 8 + w; s < n; s += (uint64_t)gridDim.x * 8) {
        if (lane < 24) hist[w][lane] = 0;
        __syncwarp();
        const uint64_t b = offs[s], e = offs[s + 1];
        const uint64_t len = e - b;
        uint32_t lc = 0;
        for (uint64_t i = b + lane; i < e; i += 32) {
            const uint32_t c = codes[i];
            atomicAdd(&hist[w][c < 24 ? c : 23], 1u);
            if (i + 12 <= e) {
                uint32_t seen = 0;
                for (int k = 0; k < 12; k++) seen |= 1u << min((uint32_t)codes[i + k], 23u);
                lc += __popc(seen) <= 4;
            }
        }
        lc = __reduce_add_sync(0xffffffffu, lc);
        __syncwarp();
        if (lane == 0) {
            float ent = 0.f, mx = 0.f;
            uint32_t std20 = 0;
            for (int c = 0; c < 20; c++) std20 += hist[w][c];
            for (int c = 0; c < 20; c++) {
                if (!hist[w][c]) continue;
                const float p = (float)hist[w][c] / (float)std20;
                ent -= p * log2f(p);
                mx = fmaxf(mx, p);
            }
            const float nl = len ? (float)len : 1.f;
            const float win = len >= 12 ? (float)(len - 11) : 1.f;
            out[s] = make_float4(ent, (float)lc / win, mx, (float)(len - std20) / nl);
        }
        __syncwarp();
    }
}

// ---- per-region features ------------------------------------------------------
struct RegionFeatArgs {
    const saber_region* reg;
    const uint4* rstat;       // HSPs, score sum, seed hits
    const uint32_t* rquery;   // query of each region (batch index)
    const uint32_t* rrank;    // rank of the region within its query (region order)
    const float4* qinfo;      // per query: length, region threshold, top best, regions
    const float4* qfeat;      // per query sequence features
    const float4* sfeat;      // per subject sequence features
    const uint64_t* soffs;    // subject offsets
    float lambda, logk;
    uint64_t n;
    float* X;                 // n x 32
};

__global__ void k_region_feats(RegionFeatArgs a) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (uint64_t)gridDim.x * blockDim.x) {
        const saber_region r = a.reg[i];
        const uint4 st = a.rstat[i];
        const uint32_t q = a.rquery[i];
        const float4 qi = a.qinfo[q];
        const float qlen = fmaxf(qi.x, 1.f), thr = fmaxf(qi.y, 1.f), top = fmaxf(qi.z, 1.f), nreg = qi.w;
        const float slen = fmaxf((float)(a.soffs[r.subject + 1] - a.soffs[r.subject]), 1.f);
        const float best = (float)r.best, spread = (float)(r.d_max - r.d_min);
        const float nh = (float)st.x, ssum = (float)st.y, hits = (float)st.z;
        const float dmid = 0.5f * (float)(r.d_min + r.d_max);
        const float ov = fmaxf(fminf(qlen, slen - dmid) - fmaxf(0.f, -dmid), 0.f);
        const float4 qf = a.qfeat[q], sf = a.sfeat[r.subject];
        float f[kTIn];
        f[0] = best / 100.f;
        f[1] = log2f(1.f + fmaxf(best, 0.f));
        f[2] = best / thr;
        f[3] = (a.lambda * best - a.logk) / 0.69314718f / 100.f;
        f[4] = (a.lambda * best - a.logk - logf(qlen) - logf(slen)) / 2.30258509f / 10.f;
        f[5] = log2f(1.f + nh);
        f[6] = log2f(1.f + hits);
        f[7] = nh > 0.f ? ssum / (100.f * nh) : 0.f;
        f[8] = log2f(1.f + ssum);
        f[9] = log2f(1.f + fmaxf(spread, 0.f));
        f[10] = spread / qlen;
        f[11] = log2f(qlen);
        f[12] = log2f(slen);
        f[13] = log2f(qlen) - log2f(slen);
        f[14] = ov / fminf(qlen, slen);
        f[15] = log2f(1.f + (float)a.rrank[i]);
        f[16] = best / top;
        f[17] = log2f(1.f + nreg);
        f[18] = qf.x;
        f[19] = qf.y;
        f[20] = qf.z;
        f[21] = sf.x;
        f[22] = sf.y;
        f[23] = sf.z;
        for (int k = kTFeat; k < kTIn; k++) f[k] = 0.f;
        float4* o = reinterpret_cast<float4*>(a.X + i * kTIn);
        for (int k = 0; k < kTIn / 4; k++) o[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
    }
}

// ---- training GEMMs: fp32 FMA on 64 x 64 tiles -----------------------------------
// C[m][n] = sum_k A[m][k] B[k][n], 256 threads, 4 x 4 outputs each, k in
// steps of 32: both operands are staged k-major in shared memory (pitch 68:
// 16-byte rows, so a thread reads its four rows and four columns of a k with
// two 128-bit loads per 16 FMA), the next step's global loads are in flight
// while a step computes.  fp32 throughout: the gradients keep the accuracy of
// a plain fp32 sum (the bf16 tensor path would round the activations).
// An operand is a loader: ld() reads a thread's 8 values of a step into
// registers, st() stores them k-major.  Loaders zero what lies outside the
// matrix.  The weight gradients contract over the batch's rows: the rows are
// split over blockIdx.z, each split writes its own partial gradient, and
// k_sum_splits adds them (2,048 rows: 16 splits x 16 tiles instead of 16
// blocks walking all rows).  A call of 2,048 rows takes eight launches and 141
// us on one GB300 (sixteen launches and 1.49 ms with one block per output
// tile, separate column sums and buffers allocated per call); its error
// against 64 bits fell from 6e-7 to 8e-8.
constexpr int kBT = 64, kBK = 32, kPitch = kBT + 4;

__device__ __forceinline__ float4 bf4(uint2 v) {
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&v.x), b = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
    return make_float4(__bfloat162float(a.x), __bfloat162float(a.y), __bfloat162float(b.x), __bfloat162float(b.y));
}

// rows r0 .. of a row-major [rows][ld] matrix, k along the columns:
// thread t takes row t / 4 and k = 4 (t % 4) + {0..3, 16..19}
struct RowsF32 {
    const float* p;
    int rows, ld;
    float4 v[2];
    __device__ __forceinline__ void load(int r0, int k0, int) {
        const int r = r0 + (threadIdx.x >> 2), k = k0 + 4 * (threadIdx.x & 3);
#pragma unroll
        for (int h = 0; h < 2; h++)
            v[h] = r < rows ? *reinterpret_cast<const float4*>(p + (size_t)r * ld + k + 16 * h)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ void store(float (*S)[kPitch]) const {
        const int r = threadIdx.x >> 2, k = 4 * (threadIdx.x & 3);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            S[k + 16 * h][r] = v[h].x;
            S[k + 16 * h + 1][r] = v[h].y;
            S[k + 16 * h + 2][r] = v[h].z;
            S[k + 16 * h + 3][r] = v[h].w;
        }
    }
};
// the same over a bf16 matrix with all its rows present
struct RowsBf16 {
    const __nv_bfloat16* p;
    int ld;
    float4 v[2];
    __device__ __forceinline__ void load(int r0, int k0, int) {
        const int r = r0 + (threadIdx.x >> 2), k = k0 + 4 * (threadIdx.x & 3);
#pragma unroll
        for (int h = 0; h < 2; h++) v[h] = bf4(*reinterpret_cast<const uint2*>(p + (size_t)r * ld + k + 16 * h));
    }
    __device__ __forceinline__ void store(float (*S)[kPitch]) const { RowsF32{nullptr, 0, 0, {v[0], v[1]}}.store(S); }
};
// the output layer's backward, dH2[i][j] = dz[i] W3[j] (H2[i][j] > 0), rows i
struct RowsDH2 {
    const float *H2, *dz;
    const __nv_bfloat16* w3;
    int rows;
    float4 v[2];
    __device__ __forceinline__ void load(int r0, int k0, int) {
        const int r = r0 + (threadIdx.x >> 2), k = k0 + 4 * (threadIdx.x & 3);
        const float d = r < rows ? dz[r] : 0.f;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float4 a = r < rows ? *reinterpret_cast<const float4*>(H2 + (size_t)r * kTHid + k + 16 * h)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 w = bf4(*reinterpret_cast<const uint2*>(w3 + k + 16 * h));
            v[h] = make_float4(a.x > 0.f ? d * w.x : 0.f, a.y > 0.f ? d * w.y : 0.f, a.z > 0.f ? d * w.z : 0.f,
                               a.w > 0.f ? d * w.w : 0.f);
        }
    }
    __device__ __forceinline__ void store(float (*S)[kPitch]) const { RowsF32{nullptr, 0, 0, {v[0], v[1]}}.store(S); }
};
// k along the rows of a row-major [..][ld] matrix, columns c0 .. c0 + 63 (those
// below cols): thread t takes columns 4 (t % 16) .. + 3 of rows t / 16 and + 16
struct ColsF32 {
    const float* p;
    int ld, cols;
    float4 v[2];
    __device__ __forceinline__ void load(int c0, int k0, int kend) {
        const int c = c0 + 4 * (threadIdx.x & 15);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int k = k0 + (threadIdx.x >> 4) + 16 * h;
            v[h] = k < kend && c < cols ? *reinterpret_cast<const float4*>(p + (size_t)k * ld + c)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void store(float (*S)[kPitch]) const {
#pragma unroll
        for (int h = 0; h < 2; h++)
            *reinterpret_cast<float4*>(&S[(threadIdx.x >> 4) + 16 * h][4 * (threadIdx.x & 15)]) = v[h];
    }
};
struct ColsBf16 {
    const __nv_bfloat16* p;
    float4 v[2];
    __device__ __forceinline__ void load(int c0, int k0, int) {
        const int c = c0 + 4 * (threadIdx.x & 15);
#pragma unroll
        for (int h = 0; h < 2; h++)
            v[h] = bf4(*reinterpret_cast<const uint2*>(p + (size_t)(k0 + (threadIdx.x >> 4) + 16 * h) * kTHid + c));
    }
    __device__ __forceinline__ void store(float (*S)[kPitch]) const { ColsF32{nullptr, 0, 0, {v[0], v[1]}}.store(S); }
};
// dH2 with k along the rows; keeps the column sums of dH2 (db2) and of
// H2 dz (dW3) of the rows this thread loads
struct ColsDH2 {
    const float *H2, *dz;
    const __nv_bfloat16* w3;
    float4 v[2];
    float4 sb, sw;
    float sz;
    __device__ __forceinline__ void load(int c0, int k0, int kend) {
        const int c = c0 + 4 * (threadIdx.x & 15);
        const float4 w = bf4(*reinterpret_cast<const uint2*>(w3 + c));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int k = k0 + (threadIdx.x >> 4) + 16 * h;
            const float d = k < kend ? dz[k] : 0.f;
            const float4 a = k < kend ? *reinterpret_cast<const float4*>(H2 + (size_t)k * kTHid + c)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            v[h] = make_float4(a.x > 0.f ? d * w.x : 0.f, a.y > 0.f ? d * w.y : 0.f, a.z > 0.f ? d * w.z : 0.f,
                               a.w > 0.f ? d * w.w : 0.f);
            sb = make_float4(sb.x + v[h].x, sb.y + v[h].y, sb.z + v[h].z, sb.w + v[h].w);
            sw = make_float4(fmaf(a.x, d, sw.x), fmaf(a.y, d, sw.y), fmaf(a.z, d, sw.z), fmaf(a.w, d, sw.w));
            sz += d;
        }
    }
    __device__ __forceinline__ void store(float (*S)[kPitch]) const { ColsF32{nullptr, 0, 0, {v[0], v[1]}}.store(S); }
};

template <class LA, class LB>
__device__ __forceinline__ void gemm_tile(LA& la, LB& lb, int m0, int n0, int kbeg, int kend, float (*As)[kPitch],
                                          float (*Bs)[kPitch], float (&acc)[4][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
    la.load(m0, kbeg, kend);
    lb.load(n0, kbeg, kend);
    for (int k0 = kbeg; k0 < kend; k0 += kBK) {
        la.store(As);
        lb.store(Bs);
        __syncthreads();
        if (k0 + kBK < kend) {
            la.load(m0, k0 + kBK, kend);
            lb.load(n0, k0 + kBK, kend);
        }
#pragma unroll
        for (int k = 0; k < kBK; k++) {
            const float4 a = *reinterpret_cast<const float4*>(&As[k][4 * ty]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[k][4 * tx]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
}

// H = relu(A W + b), A [rows][lda] fp32, W [K][256] bf16
__global__ void __launch_bounds__(256) k_layer(const float* __restrict__ A, int rows, int K,
                                               const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
                                               float* __restrict__ H) {
    __shared__ __align__(16) float As[kBK][kPitch], Bs[kBK][kPitch];
    float acc[4][4];
    const int n0 = blockIdx.x * kBT, m0 = blockIdx.y * kBT;
    RowsF32 la{A, rows, K, {}};
    ColsBf16 lb{W, {}};
    gemm_tile(la, lb, m0, n0, 0, K, As, Bs, acc);
    const int n = n0 + 4 * (threadIdx.x & 15);
    const float4 b = make_float4(bias[n], bias[n + 1], bias[n + 2], bias[n + 3]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + 4 * (threadIdx.x >> 4) + i;
        if (m < rows)
            *reinterpret_cast<float4*>(H + (size_t)m * kTHid + n) =
                make_float4(fmaxf(acc[i][0] + b.x, 0.f), fmaxf(acc[i][1] + b.y, 0.f), fmaxf(acc[i][2] + b.z, 0.f),
                            fmaxf(acc[i][3] + b.w, 0.f));
    }
}

// dH1 = (dH2 W2^T) * relu'(H1), dH2 formed from H2, dz and W3 as it is loaded
__global__ void __launch_bounds__(256) k_back_hidden(const float* __restrict__ H2, const float* __restrict__ dz,
                                                     const __nv_bfloat16* __restrict__ w3, int rows,
                                                     const __nv_bfloat16* __restrict__ W2,
                                                     const float* __restrict__ H1, float* __restrict__ dH1) {
    __shared__ __align__(16) float As[kBK][kPitch], Bs[kBK][kPitch];
    float acc[4][4];
    const int n0 = blockIdx.x * kBT, m0 = blockIdx.y * kBT;
    RowsDH2 la{H2, dz, w3, rows, {}};
    RowsBf16 lb{W2, kTHid, {}};
    gemm_tile(la, lb, m0, n0, 0, kTHid, As, Bs, acc);
    const int n = n0 + 4 * (threadIdx.x & 15);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + 4 * (threadIdx.x >> 4) + i;
        if (m >= rows) continue;
        const float4 h = *reinterpret_cast<const float4*>(H1 + (size_t)m * kTHid + n);
        *reinterpret_cast<float4*>(dH1 + (size_t)m * kTHid + n) =
            make_float4(h.x > 0.f ? acc[i][0] : 0.f, h.y > 0.f ? acc[i][1] : 0.f, h.z > 0.f ? acc[i][2] : 0.f,
                        h.w > 0.f ? acc[i][3] : 0.f);
    }
}

// Sum of a per-thread float4 over the 16 threads of a column group (threads
// t, t + 16, ...), through shared memory; valid in the first 16 threads.
__device__ __forceinline__ float4 sum_column_group(float4 v, float4* buf) {
    __syncthreads();
    buf[threadIdx.x] = v;
    __syncthreads();
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x < 16)
        for (int i = 0; i < 16; i++) {
            const float4 x = buf[threadIdx.x + 16 * i];
            s = make_float4(s.x + x.x, s.y + x.y, s.z + x.z, s.w + x.w);
        }
    return s;
}

// Partial weight gradients of the rows of split blockIdx.z into part + split *
// kOffMu (model layout).  blockIdx.y < 4: tile row blockIdx.y of dW2 = H1^T
// dH2, the first with db2, dW3 and db3; blockIdx.y == 4: dW1 = Xn^T dH1 with
// db1.
__global__ void __launch_bounds__(256) k_weight_grads(const float* __restrict__ Xn, const float* __restrict__ H1,
                                                      const float* __restrict__ H2, const float* __restrict__ dz,
                                                      const __nv_bfloat16* __restrict__ w3,
                                                      const float* __restrict__ dH1, int rows, int per_split,
                                                      float* __restrict__ part) {
    __shared__ __align__(16) float As[kBK][kPitch], Bs[kBK][kPitch];
    const int n0 = blockIdx.x * kBT, kbeg = blockIdx.z * per_split, kend = min(rows, kbeg + per_split);
    const int n = n0 + 4 * (threadIdx.x & 15);
    float* g = part + (size_t)blockIdx.z * kOffMu;
    float acc[4][4];
    float4* buf = reinterpret_cast<float4*>(&As[0][0]);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto put4 = [](float* p, float4 v) {  // model offsets of W3 and the biases are not all 16-byte aligned
        p[0] = v.x;
        p[1] = v.y;
        p[2] = v.z;
        p[3] = v.w;
    };
    if (blockIdx.y < 4) {
        const int m0 = blockIdx.y * kBT;
        ColsF32 la{H1, kTHid, kTHid, {}};
        ColsDH2 lb{H2, dz, w3, {}, zero, zero, 0.f};
        gemm_tile(la, lb, m0, n0, kbeg, kend, As, Bs, acc);
#pragma unroll
        for (int i = 0; i < 4; i++)
            put4(g + kOffW2 + (size_t)(m0 + 4 * (threadIdx.x >> 4) + i) * kTHid + n,
                 make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
        if (blockIdx.y == 0) {
            const float4 b = sum_column_group(lb.sb, buf), w = sum_column_group(lb.sw, buf);
            const float4 z = sum_column_group(make_float4(lb.sz, 0.f, 0.f, 0.f), buf);
            if (threadIdx.x < 16) {
                put4(g + kOffB2 + n, b);
                put4(g + kOffW3 + n, w);
                if (n == 0) g[kOffB3] = z.x;
            }
        }
    } else {
        ColsF32 la{Xn, kTIn, kTIn, {}};
        ColsF32 lb{dH1, kTHid, kTHid, {}};
        // column sums of dH1 beside the product: rows of the staged tiles
        float4 sb = zero;
        struct Summed {
            ColsF32& l;
            float4& s;
            __device__ __forceinline__ void load(int c0, int k0, int ke) {
                l.load(c0, k0, ke);
#pragma unroll
                for (int h = 0; h < 2; h++)
                    s = make_float4(s.x + l.v[h].x, s.y + l.v[h].y, s.z + l.v[h].z, s.w + l.v[h].w);
            }
            __device__ __forceinline__ void store(float (*S)[kPitch]) const { l.store(S); }
        } ls{lb, sb};
        gemm_tile(la, ls, 0, n0, kbeg, kend, As, Bs, acc);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int m = 4 * (threadIdx.x >> 4) + i;
            if (m < kTIn) put4(g + kOffW1 + (size_t)m * kTHid + n, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
        }
        const float4 b = sum_column_group(sb, buf);
        if (threadIdx.x < 16) put4(g + kOffB1 + n, b);
    }
}

// grad = sum over the splits (zero for the normalisation entries, which are
// not trained)
__global__ void k_sum_splits(const float* __restrict__ part, int splits, float* __restrict__ grad) {
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < kModelFloats; t += (size_t)gridDim.x * blockDim.x) {
        float s = 0.f;
        if (t < kOffMu)
            for (int k = 0; k < splits; k++) s += part[(size_t)k * kOffMu + t];
        grad[t] = s;
    }
}

// normalised inputs: Xn = (X - mu) * isd
__global__ void k_normalize(const float* __restrict__ X, uint64_t n, const float* __restrict__ model,
                            float* __restrict__ Xn) {
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * kTIn; t += (uint64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % kTIn);
        Xn[t] = k < kTFeat ? (X[t] - model[kOffMu + k]) * model[kOffIsd + k] : 0.f;
    }
}

__global__ void k_to_bf16(const float* __restrict__ src, uint64_t n, __nv_bfloat16* __restrict__ dst) {
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x)
        dst[t] = __float2bfloat16_rn(src[t]);
}

// Output layer and binary cross-entropy on its logits, positives weighted by
// pos_weight, mean over the batch: z = H2 W3 + b3, dz = w (sigmoid(z) - y) / n;
// loss accumulated in double.  A block stages 32 rows in shared memory and a
// lane sums a row's products in column order (the logit's rounding does not
// depend on the batch, so neither does the loss).
constexpr int kBceRows = 32;
__global__ void __launch_bounds__(256) k_out_bce(const float* __restrict__ H2, const __nv_bfloat16* __restrict__ w3,
                                                 const float* __restrict__ b3, const uint8_t* __restrict__ y, int n,
                                                 float pos_weight, float* __restrict__ dz, double* __restrict__ loss) {
    __shared__ float rows[kBceRows][kTHid + 1], w[kTHid];
    const int r0 = blockIdx.x * kBceRows;
    for (int t = threadIdx.x; t < kBceRows * kTHid / 4; t += 256) {
        const int r = t / (kTHid / 4), c = 4 * (t % (kTHid / 4));
        if (r0 + r >= n) break;
        const float4 v = *reinterpret_cast<const float4*>(H2 + (size_t)(r0 + r) * kTHid + c);
        rows[r][c] = v.x;
        rows[r][c + 1] = v.y;
        rows[r][c + 2] = v.z;
        rows[r][c + 3] = v.w;
    }
    w[threadIdx.x] = __bfloat162float(w3[threadIdx.x]);
    __syncthreads();
    if (threadIdx.x >= kBceRows) return;
    const int i = r0 + threadIdx.x;
    double l = 0.0;
    if (i < n) {
        float s = 0.f;
#pragma unroll 16
        for (int k = 0; k < kTHid; k++) s = fmaf(rows[threadIdx.x][k], w[k], s);
        const float zi = s + b3[0];
        const float yi = y[i] ? 1.f : 0.f;
        const float wt = y[i] ? pos_weight : 1.f;
        const float p = 1.f / (1.f + expf(-zi));
        dz[i] = wt * (p - yi) / (float)n;
        // log(1 + exp(-|z|)) + max(z, 0) - y z
        const float li = log1pf(expf(-fabsf(zi))) + fmaxf(zi, 0.f) - yi * zi;
        l = (double)(wt * li) / n;
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (threadIdx.x == 0) atomicAdd(loss, l);
}

// Adam (bias-corrected), fp32 masters, weights only (the normalisation
// entries mu / isd are not trained)
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       uint64_t n, float lr, float b1, float b2, float eps, float c1, float c2, float wd) {
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
        if (t >= kOffMu) continue;
        const float gt = g[t] + wd * w[t];
        const float mt = b1 * m[t] + (1.f - b1) * gt;
        const float vt = b2 * v[t] + (1.f - b2) * gt * gt;
        m[t] = mt;
        v[t] = vt;
        w[t] -= lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    }
}

// (x, y) -> packed bf16 pairs hi and lo with x ~ hi.x + lo.x, y ~ hi.y + lo.y
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __bfloat162float(h.x), y - __bfloat162float(h.y));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// ---- fused inference on tcgen05 -------------------------------------------------
// The weights are bf16 already; the activations (the normalised inputs and the
// layer-1 outputs) are fp32 and enter as a bf16 pair hi + lo (lo = the rounding
// residual), two products per tile with fp32 accumulation, so the result
// matches the fp32-activation forward pass of training to about 2^-16 relative.
// One persistent block per SM, tiles of 128 rows, the weights resident in
// shared memory, both layers' accumulators (128 x 256 fp32 each) in the SM's
// 512 TMEM columns.
//   layer 1: A = [hi | lo] (128 x 64), B = [W1; W1]: four MMAs of K = 16
//   layer 2: the hidden units in four chunks of 64; a chunk's accumulators are
//            read back, biased, clamped and split into hi and lo operand tiles
//            (two buffers, so that the next chunk is converted while eight
//            MMAs of this one run)
//   layer 3: each thread dots half a row of layer 2 with W3
// Operand tiles are K-major with the 128-byte swizzle: row r, 16-byte piece j
// at 128 r + 16 (j ^ (r & 7)), 64 values of K a row.
//
// One GB300, a call from host rows (an mma.sync m16n8k16 kernel, 16 rows a warp
// with the weight fragments read from L1 -> this one): 200 rows 113 -> 69 us,
// 20,000 153 -> 109, 1 M 1633 -> 1154 us, of which the rows' copy to the device
// is about 750.
//
// Every wait on an mbarrier is bounded: when one runs out the block sets *err,
// stops waiting, still finishes its loop and frees its TMEM, and the host
// reports the error.
constexpr int kMtRows = 128, kMtThreads = 256;
constexpr uint32_t kMtTile = 128 * 128;          // bytes of a 128 x 64 bf16 operand tile
constexpr uint32_t kMtW2 = 0;                    // four 256 x 64 tiles of W2^T
constexpr uint32_t kMtW1 = kMtW2 + 4 * 2 * kMtTile;
constexpr uint32_t kMtA = kMtW1 + 2 * kMtTile;   // two buffers of (hi, lo); the layer-1 operand uses the second
constexpr size_t kMtSmem = kMtA + 4 * kMtTile + 1024;  // + room to align the base to 1024 bytes
constexpr uint32_t kMtIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t mt_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory descriptor of a K-major tile, 128-byte swizzle, groups of eight
// rows 1024 bytes apart.
__device__ __forceinline__ uint64_t mt_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mt_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(d), "l"(a), "l"(b), "r"(kMtIdesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mt_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" : : "r"(bar) : "memory");
}

// Waits for the phase of parity `phase`; false when it does not come.
__device__ __forceinline__ bool mt_wait(uint32_t bar, uint32_t phase) {
    for (int i = 0; i < (1 << 15); i++) {  // (a try lasts two microseconds at most)
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(phase), "r"(2000u)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// 32 columns of this thread's TMEM lane.
__device__ __forceinline__ void mt_ld32(uint32_t (&v)[32], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void mt_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mt_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__global__ void __launch_bounds__(kMtThreads, 1) k_mlp_tc(const float* __restrict__ X, uint64_t n,
                                                          const float* __restrict__ model,
                                                          const __nv_bfloat16* __restrict__ wb,
                                                          float* __restrict__ logit, uint32_t* __restrict__ err) {
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t bars[3];  // chunk buffers 0 and 1, layer 1
    __shared__ uint32_t tmem_at;
    __shared__ float norm[2 * kTIn], half_dot[kMtRows];
    uint8_t* base = raw + ((1024u - (mt_smem(raw) & 1023u)) & 1023u);
    const uint32_t sb = mt_smem(base);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned short* w = reinterpret_cast<const unsigned short*>(wb);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" : : "r"(mt_smem(&tmem_at)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32)
        for (int i = 0; i < 3; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(mt_smem(&bars[i])) : "memory");
    if (tid < 2 * kTIn) norm[tid] = model[kOffMu + tid];  // mu, then isd
    // weights, transposed to rows of the output unit: W2 in four tiles of 64
    // inputs, W1 twice in one
    for (int t = tid; t < 40 * kTHid; t += kMtThreads) {
        const int o = t & (kTHid - 1), p = t >> 8;  // output unit, piece of eight inputs
        const bool l2 = p < 32;
        const unsigned short* src = w + (l2 ? kOffW2 + (size_t)p * 8 * kTHid : kOffW1 + (size_t)(p & 3) * 8 * kTHid) + o;
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = (uint32_t)src[2 * i * kTHid] | ((uint32_t)src[(2 * i + 1) * kTHid] << 16);
        const int j = p & 7;
        uint8_t* dst = base + (l2 ? kMtW2 + (uint32_t)(p >> 3) * 2 * kMtTile : kMtW1) + 128 * o + 16 * (j ^ (o & 7));
        *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mt_before_sync();
    __syncthreads();
    mt_after_sync();
    const uint32_t tmem = tmem_at;
    const uint32_t d1 = tmem, d2 = tmem + 256;
    const uint32_t lanes = (uint32_t)(warp & 3) * 32u << 16;  // this warp's TMEM lanes
    const int row = (warp & 3) * 32 + lane, hf = warp >> 2;   // its row of the tile, its half of the columns
    const uint32_t bar0 = mt_smem(&bars[0]), bar1 = mt_smem(&bars[1]), barL = mt_smem(&bars[2]);
    uint32_t ph0 = 0, ph1 = 0, phL = 0;
    bool dead = false;
    const uint64_t tiles = (n + kMtRows - 1) / kMtRows;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        // layer-1 operand: two threads per row, 16 features each
        {
            const int r = tid >> 1, h = tid & 1;
            const uint64_t gr = tile * kMtRows + r;
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float4 x = gr < n ? __ldg(reinterpret_cast<const float4*>(X + gr * kTIn + 16 * h) + q)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
                const int k = 16 * h + 4 * q;
                float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int e = 0; e < 4; e++) v[e] = gr < n && k + e < kTFeat ? (v[e] - norm[k + e]) * norm[kTIn + k + e] : 0.f;
                split2(v[0], v[1], hi[2 * q], lo[2 * q]);
                split2(v[2], v[3], hi[2 * q + 1], lo[2 * q + 1]);
            }
            uint8_t* a1 = base + kMtA + 2 * kMtTile + 128 * r;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                *reinterpret_cast<uint4*>(a1 + 16 * ((2 * h + q) ^ (r & 7))) =
                    make_uint4(hi[4 * q], hi[4 * q + 1], hi[4 * q + 2], hi[4 * q + 3]);
                *reinterpret_cast<uint4*>(a1 + 16 * ((4 + 2 * h + q) ^ (r & 7))) =
                    make_uint4(lo[4 * q], lo[4 * q + 1], lo[4 * q + 2], lo[4 * q + 3]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mt_before_sync();
        __syncthreads();
        if (tid == 0) {
            mt_after_sync();
#pragma unroll
            for (int k = 0; k < 4; k++)
                mt_mma(d1, mt_desc(sb + kMtA + 2 * kMtTile + 32 * k), mt_desc(sb + kMtW1 + 32 * k), k > 0);
            mt_commit(barL);
        }
        if (!dead) dead = !mt_wait(barL, phL);
        phL ^= 1u;
        mt_after_sync();
#pragma unroll 1
        for (int c = 0; c < 4; c++) {
            // the buffer's last MMAs (chunk c - 2) are done before it is written
            if (c >= 2) {
                if (c & 1) {
                    if (!dead) dead = !mt_wait(bar1, ph1);
                    ph1 ^= 1u;
                } else {
                    if (!dead) dead = !mt_wait(bar0, ph0);
                    ph0 ^= 1u;
                }
            }
            uint32_t v[32];
            const int col = 64 * c + 32 * hf;
            mt_ld32(v, d1 + lanes + (uint32_t)col);
            uint8_t* ah = base + kMtA + (uint32_t)(c & 1) * 2 * kMtTile + 128 * row;
            uint8_t* al = ah + kMtTile;
#pragma unroll
            for (int q = 0; q < 4; q++) {  // eight units: one 16-byte piece of hi and of lo
                const float4 b0 = __ldg(reinterpret_cast<const float4*>(model + kOffB1 + col + 8 * q));
                const float4 b1 = __ldg(reinterpret_cast<const float4*>(model + kOffB1 + col + 8 * q + 4));
                const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; e++)
                    split2(fmaxf(__uint_as_float(v[8 * q + 2 * e]) + bb[2 * e], 0.f),
                           fmaxf(__uint_as_float(v[8 * q + 2 * e + 1]) + bb[2 * e + 1], 0.f), hi[e], lo[e]);
                const int j = (4 * hf + q) ^ (row & 7);
                *reinterpret_cast<uint4*>(ah + 16 * j) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(al + 16 * j) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mt_before_sync();
            __syncthreads();
            if (tid == 0) {
                mt_after_sync();
                const uint32_t a0 = sb + kMtA + (uint32_t)(c & 1) * 2 * kMtTile, b0 = sb + kMtW2 + (uint32_t)c * 2 * kMtTile;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    mt_mma(d2, mt_desc(a0 + 32 * k), mt_desc(b0 + 32 * k), c > 0 || k > 0);
                    mt_mma(d2, mt_desc(a0 + kMtTile + 32 * k), mt_desc(b0 + 32 * k), 1u);
                }
                mt_commit(c & 1 ? bar1 : bar0);
            }
        }
        if (!dead) dead = !mt_wait(bar0, ph0);
        ph0 ^= 1u;
        if (!dead) dead = !mt_wait(bar1, ph1);
        ph1 ^= 1u;
        mt_after_sync();
        // layer 3: this thread's 128 columns of its row
        float sum = 0.f;
#pragma unroll 1
        for (int c = 0; c < 4; c++) {
            uint32_t v[32];
            const int col = 128 * hf + 32 * c;
            mt_ld32(v, d2 + lanes + (uint32_t)col);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float4 b = __ldg(reinterpret_cast<const float4*>(model + kOffB2 + col + 4 * q));
                const float4 w3 = bf4(__ldg(reinterpret_cast<const uint2*>(wb + kOffW3 + col + 4 * q)));
                sum = fmaf(fmaxf(__uint_as_float(v[4 * q]) + b.x, 0.f), w3.x, sum);
                sum = fmaf(fmaxf(__uint_as_float(v[4 * q + 1]) + b.y, 0.f), w3.y, sum);
                sum = fmaf(fmaxf(__uint_as_float(v[4 * q + 2]) + b.z, 0.f), w3.z, sum);
                sum = fmaf(fmaxf(__uint_as_float(v[4 * q + 3]) + b.w, 0.f), w3.w, sum);
            }
        }
        if (hf) half_dot[row] = sum;
        mt_before_sync();
        __syncthreads();
        mt_after_sync();
        const uint64_t gr = tile * kMtRows + row;
        if (!hf && gr < n) logit[gr] = sum + half_dot[row] + model[kOffB3];
    }
    if (dead) atomicExch(err, 1u);
    mt_before_sync();
    __syncthreads();
    if (warp == 0) {
        mt_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" : : "r"(tmem) : "memory");
    }
}

__global__ void k_gather_rows(const float* __restrict__ Xn, const uint8_t* __restrict__ y,
                              const uint32_t* __restrict__ idx, int nb, float* __restrict__ Xb, uint8_t* __restrict__ yb) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nb * kTIn; t += gridDim.x * blockDim.x) {
        const int i = t / kTIn, k = t % kTIn;
        Xb[t] = Xn[(size_t)idx[i] * kTIn + k];
        if (k == 0) yb[i] = y[idx[i]];
    }
}

// ---- host side -------------------------------------------------------------------
int triage_upload_model(saber_gpu* h, DevBuf& model, DevBuf& wb, const float* host_model);
static int upload_model(saber_gpu* h, DevBuf& model, DevBuf& wb, const float* host_model) {
    return triage_upload_model(h, model, wb, host_model);
}

int triage_upload_model(saber_gpu* h, DevBuf& model, DevBuf& wb, const float* host_model) {
    CUALLOC(h, model, kModelFloats * 4);
    CUALLOC(h, wb, kModelFloats * 2);
    CU(h, cudaMemcpyAsync(model.p, host_model, kModelFloats * 4, cudaMemcpyHostToDevice, h->stream));
    k_to_bf16<<<nblocks(kModelFloats, 256), 256, 0, h->stream>>>(model.as<float>(), kModelFloats,
                                                                 wb.as<__nv_bfloat16>());
    CU(h, cudaGetLastError());
    return SABER_OK;
}

// Row splits of the weight gradients: at least 128 rows each, at most 32 (the
// partials stay under 10 MB and are added from L2).
static int grad_splits(uint64_t n) { return (int)std::min<uint64_t>(std::max<uint64_t>(n / 128, 1), 32); }

// forward + backward of one batch (inputs already normalised in Xn, labels
// in y): gradients written to grad (model layout), loss added to *loss
static int fwd_bwd(saber_gpu* h, TriageScratch& d, int n, float pos_weight) {
    cudaStream_t s = h->stream;
    const float* mdl = d.model.as<float>();
    const __nv_bfloat16* wb = d.wb.as<__nv_bfloat16>();
    const float* Xn = d.Xn.as<float>();
    float* H1 = d.H1.as<float>();
    float* H2 = d.H2.as<float>();
    float* dz = d.dz.as<float>();
    const dim3 tiles(kTHid / kBT, (unsigned)((n + kBT - 1) / kBT));
    k_layer<<<tiles, 256, 0, s>>>(Xn, n, kTIn, wb + kOffW1, mdl + kOffB1, H1);
    k_layer<<<tiles, 256, 0, s>>>(H1, n, kTHid, wb + kOffW2, mdl + kOffB2, H2);
    k_out_bce<<<(unsigned)((n + kBceRows - 1) / kBceRows), 256, 0, s>>>(
        H2, wb + kOffW3, mdl + kOffB3, d.y.as<uint8_t>(), n, pos_weight, dz, d.loss.as<double>());
    k_back_hidden<<<tiles, 256, 0, s>>>(H2, dz, wb + kOffW3, n, wb + kOffW2, H1, d.dH1.as<float>());
    int splits = grad_splits((uint64_t)n);
    const int per = (((n + splits - 1) / splits) + kBK - 1) / kBK * kBK;
    splits = (n + per - 1) / per;
    k_weight_grads<<<dim3(kTHid / kBT, 5, (unsigned)splits), 256, 0, s>>>(Xn, H1, H2, dz, wb + kOffW3,
                                                                          d.dH1.as<float>(), n, per, d.part.as<float>());
    k_sum_splits<<<nblocks(kModelFloats, 256), 256, 0, s>>>(d.part.as<float>(), splits, d.grad.as<float>());
    CU(h, cudaGetLastError());
    return SABER_OK;
}

static int reserve_batch(saber_gpu* h, TriageScratch& d, uint64_t n) {
    CUALLOC(h, d.Xn, n * kTIn * 4);
    CUALLOC(h, d.y, n + 16);
    CUALLOC(h, d.H1, n * kTHid * 4);
    CUALLOC(h, d.H2, n * kTHid * 4);
    CUALLOC(h, d.dz, n * 4 + 16);
    CUALLOC(h, d.dH1, n * kTHid * 4);
    CUALLOC(h, d.part, (uint64_t)grad_splits(n) * kOffMu * 4);
    CUALLOC(h, d.grad, kModelFloats * 4);
    CUALLOC(h, d.loss, 16);
    return SABER_OK;
}

int triage_grads(saber_gpu* h, const float* model, const float* X, const uint8_t* y, uint32_t n, float pos_weight,
                 float* grads, double* loss) {
    if (n == 0) return fail(h, SABER_ERR_CUDA, "no rows: invalid launch configuration");
    TriageScratch& d = h->tg;
    const SpareUse use(h, kSpareTriage);
    int rc = upload_model(h, d.model, d.wb, model);
    if (rc != SABER_OK) return rc;
    rc = reserve_batch(h, d, n);
    if (rc != SABER_OK) return rc;
    cudaStream_t s = h->stream;
    CUALLOC(h, d.X, (uint64_t)n * kTIn * 4);
    CU(h, cudaMemcpyAsync(d.X.p, X, (uint64_t)n * kTIn * 4, cudaMemcpyHostToDevice, s));
    CU(h, cudaMemcpyAsync(d.y.p, y, n, cudaMemcpyHostToDevice, s));
    CU(h, cudaMemsetAsync(d.loss.p, 0, 8, s));
    k_normalize<<<nblocks((uint64_t)n * kTIn, 256), 256, 0, s>>>(d.X.as<float>(), n, d.model.as<float>(),
                                                                  d.Xn.as<float>());
    rc = fwd_bwd(h, d, (int)n, pos_weight);
    if (rc != SABER_OK) return rc;
    CU(h, cudaMemcpyAsync(grads, d.grad.p, kModelFloats * 4, cudaMemcpyDeviceToHost, s));
    double l = 0;
    CU(h, cudaMemcpyAsync(&l, d.loss.p, 8, cudaMemcpyDeviceToHost, s));
    CU(h, cudaStreamSynchronize(s));
    if (loss) *loss = l;
    return SABER_OK;
}

int triage_train(saber_gpu* h, float* model, const float* X, const uint8_t* y, uint64_t n,
                 const saber_triage_train_cfg* cfg, saber_triage_train_stats* st) {
    if (n == 0) return fail(h, SABER_ERR_ARG, "no training samples");
    cudaStream_t s = h->stream;
    const int B = (int)std::max<uint32_t>(32, cfg->batch);
    TriageScratch& d = h->tg;
    const SpareUse use(h, kSpareTriage);
    int rc = upload_model(h, d.model, d.wb, model);
    if (rc != SABER_OK) return rc;
    rc = reserve_batch(h, d, (uint64_t)B);
    if (rc != SABER_OK) return rc;
    DevBuf Xall, yall;
    CUALLOC(h, Xall, n * kTIn * 4);
    CUALLOC(h, yall, n + 16);
    CUALLOC(h, d.m, kModelFloats * 4);
    CUALLOC(h, d.v, kModelFloats * 4);
    CU(h, cudaMemcpyAsync(Xall.p, X, n * kTIn * 4, cudaMemcpyHostToDevice, s));
    CU(h, cudaMemcpyAsync(yall.p, y, n, cudaMemcpyHostToDevice, s));
    CU(h, cudaMemsetAsync(d.m.p, 0, kModelFloats * 4, s));
    CU(h, cudaMemsetAsync(d.v.p, 0, kModelFloats * 4, s));
    // normalised copy of every sample; each epoch's batches gather rows
    // through a shuffled order (seeded)
    DevBuf Xnall, didx;
    CUALLOC(h, Xnall, n * kTIn * 4);
    CUALLOC(h, didx, n * 4);
    k_normalize<<<nblocks(n * kTIn, 256), 256, 0, s>>>(Xall.as<float>(), n, d.model.as<float>(), Xnall.as<float>());
    std::vector<uint32_t> order(n);
    for (uint64_t i = 0; i < n; i++) order[i] = (uint32_t)i;
    std::mt19937_64 rng(cfg->seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    uint64_t step = 0;
    double last_loss = 0;
    for (uint32_t ep = 0; ep < cfg->epochs; ep++) {
        std::shuffle(order.begin(), order.end(), rng);
        CU(h, cudaMemcpyAsync(didx.p, order.data(), n * 4, cudaMemcpyHostToDevice, s));
        CU(h, cudaMemsetAsync(d.loss.p, 0, 8, s));
        uint32_t nb = 0;
        for (uint64_t b0 = 0; b0 < n; b0 += B) {
            const int nbat = (int)std::min<uint64_t>(B, n - b0);
            k_gather_rows<<<nblocks((uint64_t)nbat * kTIn, 256), 256, 0, s>>>(
                Xnall.as<float>(), yall.as<uint8_t>(), didx.as<uint32_t>() + b0, nbat, d.Xn.as<float>(),
                d.y.as<uint8_t>());
            rc = fwd_bwd(h, d, nbat, cfg->pos_weight);
            if (rc != SABER_OK) return rc;
            step++;
            const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);
            k_adam<<<nblocks(kModelFloats, 256), 256, 0, s>>>(d.model.as<float>(), d.grad.as<float>(), d.m.as<float>(),
                                                              d.v.as<float>(), kModelFloats, cfg->lr, b1, b2, eps, c1, c2,
                                                              cfg->weight_decay);
            k_to_bf16<<<nblocks(kModelFloats, 256), 256, 0, s>>>(d.model.as<float>(), kModelFloats,
                                                                 d.wb.as<__nv_bfloat16>());
            CU(h, cudaGetLastError());
            nb++;
        }
        double l = 0;
        CU(h, cudaMemcpyAsync(&l, d.loss.p, 8, cudaMemcpyDeviceToHost, s));
        CU(h, cudaStreamSynchronize(s));
        last_loss = nb ? l / nb : 0.0;
    }
    CU(h, cudaMemcpyAsync(model, d.model.p, kModelFloats * 4, cudaMemcpyDeviceToHost, s));
    CU(h, cudaStreamSynchronize(s));
    if (st) {
        st->steps = step;
        st->final_loss = last_loss;
    }
    return SABER_OK;
}

static int mlp_launch(saber_gpu* h, DevBuf& model, DevBuf& wb, const float* d_X, uint64_t n, float* d_logit) {
    CU(h, cudaFuncSetAttribute(k_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMtSmem));
    const unsigned grid = (unsigned)std::min<uint64_t>((n + kMtRows - 1) / kMtRows, (uint64_t)h->sm_count);
    k_mlp_tc<<<grid, kMtThreads, kMtSmem, h->stream>>>(d_X, n, model.as<float>(), wb.as<__nv_bfloat16>(), d_logit,
                                                       h->tr_err.as<uint32_t>());
    CU(h, cudaGetLastError());
    return SABER_OK;
}
static int mlp_begin(saber_gpu* h) {
    CUALLOC(h, h->tr_err, 4);
    CU(h, cudaMemsetAsync(h->tr_err.p, 0, 4, h->stream));
    return SABER_OK;
}
static int mlp_end(saber_gpu* h) {
    uint32_t e = 0;
    CU(h, cudaMemcpyAsync(&e, h->tr_err.p, 4, cudaMemcpyDeviceToHost, h->stream));
    CU(h, cudaStreamSynchronize(h->stream));
    if (e) return fail(h, SABER_ERR_DEVICE, "the triage network's matrix pipeline did not complete");
    return SABER_OK;
}

// logits of n feature rows with the installed model or the given one
int triage_predict(saber_gpu* h, DevBuf& model, DevBuf& wb, const float* d_X, uint64_t n, float* d_logit) {
    if (n == 0) return SABER_OK;
    int rc = mlp_begin(h);
    if (rc == SABER_OK) rc = mlp_launch(h, model, wb, d_X, n, d_logit);
    return rc != SABER_OK ? rc : mlp_end(h);
}

// Rows of a chunk of a host call: a chunk's copy (16 MB) runs on the handle's
// copy stream while the chunk before it is computed.  1 M rows on one GB300:
// 1154 us in one piece, 921 in eight.
constexpr uint64_t kPredictChunk = 128 << 10;

int triage_predict_host(saber_gpu* h, const float* model, const float* X, uint64_t n, float* logits) {
    TriageScratch& d = h->tg;
    const SpareUse use(h, kSpareTriage);
    int rc = upload_model(h, d.model, d.wb, model);
    if (rc != SABER_OK) return rc;
    CUALLOC(h, d.X, std::max<uint64_t>(n, 1) * kTIn * 4);
    CUALLOC(h, d.z, std::max<uint64_t>(n, 1) * 4);
    rc = mlp_begin(h);
    if (rc != SABER_OK) return rc;
    if (!h->copy_stream) {
        CU(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
        CU(h, cudaEventCreateWithFlags(&h->copy_event, cudaEventDisableTiming));
    }
    // (the buffers are the handle's, and every earlier call has waited for its
    // stream; no return leaves a copy from the caller's rows in flight)
    struct Wait {
        cudaStream_t s;
        ~Wait() { cudaStreamSynchronize(s); }
    } wait{h->copy_stream};
    for (uint64_t r = 0; r < n; r += kPredictChunk) {
        const uint64_t k = std::min<uint64_t>(kPredictChunk, n - r);
        CU(h, cudaMemcpyAsync(d.X.as<float>() + r * kTIn, X + r * kTIn, k * kTIn * 4, cudaMemcpyHostToDevice,
                              h->copy_stream));
        CU(h, cudaEventRecord(h->copy_event, h->copy_stream));
        CU(h, cudaStreamWaitEvent(h->stream, h->copy_event, 0));
        rc = mlp_launch(h, d.model, d.wb, d.X.as<float>() + r * kTIn, k, d.z.as<float>() + r);
        if (rc != SABER_OK) return rc;
    }
    CU(h, cudaMemcpyAsync(logits, d.z.p, n * 4, cudaMemcpyDeviceToHost, h->stream));
    return mlp_end(h);
}

// Region features for the engine: uploads the batch's regions and computes
// the feature rows on the device (kept in h->tr_X); sequence features of the
// database are computed once per loaded database.
int triage_region_features(saber_gpu* h, const saber_region* d_reg, const uint4* d_rstat, const uint32_t* d_rq,
                           const uint32_t* d_rrank, const float4* d_qinfo, uint64_t n, float lambda, float logk) {
    const Dataset& ds = h->main;
    const QuerySet& qs = ds.qs;
    cudaStream_t s = h->stream;
    if (!h->tr_sfeat_ok) {
        CUALLOC(h, h->tr_sfeat, std::max<uint64_t>(ds.nsub, 1) * sizeof(float4));
        if (ds.nsub)
            k_seq_feats<<<(unsigned)std::min<uint64_t>((ds.nsub + 7) / 8, 65535u * 8), 256, 0, s>>>(
                ds.res.as<uint8_t>(), ds.soff.as<uint64_t>(), ds.nsub, h->tr_sfeat.as<float4>());
        CU(h, cudaGetLastError());
        h->tr_sfeat_ok = true;
    }
    CUALLOC(h, h->tr_qfeat, std::max<uint64_t>(qs.nq, 1) * sizeof(float4));
    if (qs.nq)
        k_seq_feats<<<(unsigned)std::min<uint64_t>((qs.nq + 7) / 8, 65535u * 8), 256, 0, s>>>(
            qs.codes.as<uint8_t>(), qs.offsets.as<uint64_t>(), qs.nq, h->tr_qfeat.as<float4>());
    const uint64_t nn = std::max<uint64_t>(n, 1);
    CUALLOC(h, h->tr_X, nn * kTIn * 4);
    CUALLOC(h, h->tr_logit, nn * 4);
    RegionFeatArgs a;
    a.reg = d_reg;
    a.rstat = d_rstat;
    a.rquery = d_rq;
    a.rrank = d_rrank;
    a.qinfo = d_qinfo;
    a.qfeat = h->tr_qfeat.as<float4>();
    a.sfeat = h->tr_sfeat.as<float4>();
    a.soffs = ds.soff.as<uint64_t>();
    a.lambda = lambda;
    a.logk = logk;
    a.n = n;
    a.X = h->tr_X.as<float>();
    if (n) k_region_feats<<<nblocks(n, 256), 256, 0, s>>>(a);
    CU(h, cudaGetLastError());
    return SABER_OK;
}

}  // namespace saber
