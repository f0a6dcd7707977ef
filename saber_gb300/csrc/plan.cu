// Window plans and the two-stage banded scoring of a batch's candidate regions
// on the device: Engine::plan_windows and score_windows (src/search/engine.rs:
// 1247-1324, 1021-1099) over the regions where the scan left them, and the
// first cut of finish (engine.rs:1127-1160), so that only regions which can be
// reported reach the host.
//
// A search has up to thousands of regions per query and reports a few.  On the
// host, planning, building the jobs, the second-stage decision and the E-value
// cut each walked all of them (15 M regions of an 11,000-query batch: 40 bytes
// a region down, 32 bytes a job up, about 100 ms of host loops; a 64-query
// batch spent 2 of its 7 ms starting threads for them).  One GB300, a whole
// search, host -> device: 11,000 queries x 150 M residues 531 -> 385 ms, 64 x 6 M
// 6.6 -> 5.6 ms, 400 x 150 M bases 37.1 -> 31.9 ms.
//
// Whole-number work is the host's.  The f64 thresholds (the score that sends a
// region to the second stage, the E-value cut) are logarithms and exponentials
// whose last bits may differ from the host's libm: a stage-two decision within
// kTie of its threshold, or one that a length adjustment within kTie of a whole
// number could turn, is left to the host (all of a batch's in one exchange), and
// the cut keeps a margin (the host applies the exact rule to what it gets).
#include <cub/cub.cuh>
#include <cuda_runtime.h>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cmath>

#include "runtime.cuh"

namespace saber {

constexpr double kTie = 1e-10;        // relative to the terms summed; the two libms differ by about 1e-15 of them
constexpr double kCutMargin = 1e-7;
constexpr int64_t kBandScoreMinCells = 1 << 20;  // engine.rs:401
constexpr int64_t kBandCostRatio = 12;           // engine.rs:402
constexpr int64_t kBandBridge = 1024;            // engine.rs:404
constexpr int kPlanGroup = 64;                   // regions of one (query, subject) pair (scan's limit)

struct DevPlan {
    int32_t lo, hi, blo, bhi;
    int32_t band;  // the plan is banded
    int32_t kind;  // stage 1: 0 full window, 1 narrow band, 2 plan band
};

__global__ void k_plan_keys(const saber_region* __restrict__ reg, uint32_t n, int bs, unsigned long long* __restrict__ key,
                            uint32_t* __restrict__ idx) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const saber_region r = reg[i];
        key[i] = ((unsigned long long)r.query << bs) | r.subject;
        idx[i] = i;
    }
}

__global__ void k_plan_flags(const unsigned long long* __restrict__ key, uint32_t n, uint8_t* __restrict__ flag) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        flag[i] = i == 0 || key[i] != key[i - 1];
}

// Spans of one pair's regions, one thread per pair: the strong regions (best
// at least max(2 hsp_threshold, top / 4)) closer than kBandBridge share one
// span, the others keep their own.
__global__ void k_plan_spans(const saber_region* __restrict__ reg, const uint32_t* __restrict__ by,
                             const uint32_t* __restrict__ starts, const uint32_t* __restrict__ ngroups, uint32_t n,
                             int hsp_threshold, int2* __restrict__ span) {
    const uint32_t ng = *ngroups;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x) {
        const uint32_t a = starts[g], b = g + 1 < ng ? starts[g + 1] : n;
        if (b - a == 1) {
            const saber_region r = reg[by[a]];
            span[by[a]] = make_int2(r.d_min, r.d_max);
            continue;
        }
        int64_t top = INT64_MIN;
        for (uint32_t t = a; t < b; t++) {
            const saber_region r = reg[by[t]];
            span[by[t]] = make_int2(r.d_min, r.d_max);
            top = max(top, (int64_t)r.best);
        }
        const int64_t strong = max(2 * (int64_t)hsp_threshold, top / 4);
        // strong regions by (d_min, d_max, position): insertion into a list
        uint32_t id[kPlanGroup];
        int lo[kPlanGroup], hi[kPlanGroup];
        int m = 0;
        for (uint32_t t = a; t < b && m < kPlanGroup; t++) {
            const uint32_t i = by[t];
            const saber_region r = reg[i];
            if (r.best < strong) continue;
            int p = m++;
            while (p > 0 && (lo[p - 1] > r.d_min || (lo[p - 1] == r.d_min && hi[p - 1] > r.d_max))) {
                lo[p] = lo[p - 1];
                hi[p] = hi[p - 1];
                id[p] = id[p - 1];
                p--;
            }
            lo[p] = r.d_min;
            hi[p] = r.d_max;
            id[p] = i;
        }
        for (int s = 0; s < m;) {
            const int l = lo[s];
            int64_t h = hi[s];
            int e = s + 1;
            while (e < m && (int64_t)lo[e] - h <= kBandBridge) {
                h = max(h, (int64_t)hi[e]);
                e++;
            }
            for (int t = s; t < e; t++) span[id[t]] = make_int2(l, (int)h);
            s = e;
        }
    }
}

__device__ __forceinline__ void pl_window(int64_t slack, int64_t dmin, int64_t dmax, int64_t sl, int64_t qlen, int64_t& lo,
                                          int64_t& hi) {
    lo = min(max(dmin - slack, (int64_t)0), sl);
    hi = max(min(qlen + dmax + slack, sl), lo);
    if ((hi - lo) * 4 >= sl * 3) {
        lo = 0;
        hi = sl;
    }
}
__device__ __forceinline__ void pl_clip(int64_t& lo, int64_t& hi, int64_t m, int64_t n) {
    lo = max(lo, -(m - 1));
    hi = min(hi, n - 1);
}
__device__ __forceinline__ bool pl_covers(int64_t lo, int64_t hi, int64_t m, int64_t n) {
    return lo <= -(m - 1) && hi >= n - 1;
}

__device__ __forceinline__ saber_band_job pl_job(uint32_t q, uint32_t subject, uint64_t sbase, int64_t lo, int64_t hi,
                                                 int64_t blo, int64_t bhi) {
    saber_band_job j;
    j.query = q;
    j.subject = subject;
    j.win_begin = sbase + (uint64_t)lo;
    j.win_len = (uint32_t)(hi - lo);
    j.band_lo = (int32_t)max(min(blo, (int64_t)INT32_MAX), (int64_t)INT32_MIN);
    j.band_hi = (int32_t)max(min(bhi, (int64_t)INT32_MAX), (int64_t)INT32_MIN);
    j.flags = 0;
    return j;
}

// Plan and stage-1 job of every region.
__global__ void k_plan_jobs(const saber_region* __restrict__ reg, const int2* __restrict__ span, uint32_t n,
                            const uint64_t* __restrict__ qoffs, const uint64_t* __restrict__ soffs, PlanParams P,
                            DevPlan* __restrict__ plan, saber_band_job* __restrict__ jobs,
                            unsigned long long* __restrict__ banded) {
    unsigned long long nb = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const saber_region r = reg[i];
        const int64_t qlen = (int64_t)(qoffs[r.query + 1] - qoffs[r.query]);
        const uint64_t sbase = soffs[r.subject];
        const int64_t sl = (int64_t)(soffs[r.subject + 1] - sbase);
        int64_t lo, hi, blo = 0, bhi = 0;
        bool band = false;
        pl_window(P.window_slack, r.d_min, r.d_max, sl, qlen, lo, hi);
        if (r.best != 0) {
            const int64_t s0 = span[i].x, s1 = span[i].y;
            if (P.score_band > 0) {
                const int64_t w = P.score_band;
                lo = min(max(s0 - w, (int64_t)0), sl);
                hi = max(min(qlen + s1 + w, sl), lo);
                const int64_t nn = hi - lo;
                blo = s0 - w - lo;
                bhi = s1 + w - lo;
                pl_clip(blo, bhi, qlen, nn);
                band = !(nn == 0 || pl_covers(blo, bhi, qlen, nn));
            } else if (qlen * (hi - lo) >= kBandScoreMinCells) {
                int64_t ulo, uhi;
                pl_window(P.window_slack, s0, s1, sl, qlen, ulo, uhi);
                const int64_t nn = uhi - ulo;
                int64_t l = s0 - ulo - P.window_slack, h = s1 - ulo + P.window_slack;
                pl_clip(l, h, qlen, nn);
                if (!pl_covers(l, h, qlen, nn)) {
                    const int64_t wd = max(h - l + 1, (int64_t)0), rows = min(qlen, nn + wd);
                    if (wd * rows * kBandCostRatio < qlen * nn) {
                        lo = ulo;
                        hi = uhi;
                        blo = l;
                        bhi = h;
                        band = true;
                    }
                }
            }
        }
        DevPlan p;
        p.lo = (int32_t)lo;
        p.hi = (int32_t)hi;
        p.blo = band ? (int32_t)blo : 0;
        p.bhi = band ? (int32_t)bhi : 0;
        p.band = band;
        const int64_t nw = hi - lo;
        if (!band) {
            p.kind = 0;
            jobs[i] = pl_job(r.query, r.subject, sbase, lo, hi, -qlen, nw);
        } else {
            nb++;
            if (0 < P.prefilter_band && P.prefilter_band < P.score_band) {
                p.kind = 1;
                int64_t l = (int64_t)r.d_min - P.prefilter_band - lo, h = (int64_t)r.d_max + P.prefilter_band - lo;
                pl_clip(l, h, qlen, nw);
                jobs[i] = pl_job(r.query, r.subject, sbase, lo, hi, l, h);
            } else {
                p.kind = 2;
                jobs[i] = pl_job(r.query, r.subject, sbase, lo, hi, blo, bhi);
            }
        }
        plan[i] = p;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nb += __shfl_xor_sync(0xffffffffu, nb, o);
    if ((threadIdx.x & 31) == 0 && nb) atomicAdd(banded, nb);
}

// QueryStatistics::space_lower_bound (stats.rs) in f64: the length adjustment
// before it is rounded up, and how far it may be off; the space for one.
__device__ __forceinline__ double pl_adjustment(const PlanParams& P, int64_t qlen, int64_t sl, double& eps) {
    const double m = (double)max(qlen, (int64_t)1), n = (double)max(sl, (int64_t)1);
    const double l = log(m * n);
    eps = kTie * (fabs(P.adl) * (fabs(P.log_k) + l) + fabs(P.beta) + 1.0);
    return P.adl * (P.log_k + l) + P.beta;
}
__device__ __forceinline__ double pl_space(const PlanParams& P, int64_t qlen, int64_t sl, double up) {
    const double m = (double)max(qlen, (int64_t)1), n = (double)max(sl, (int64_t)1);
    return P.num_seqs * fmax(m - up, 1.0) * fmax(n - up, 1.0);
}

// Stage-2 decision: flag the regions whose narrow score reaches prefilter_frac
// of the floor's lower bound (floor_lower_bound, stats.rs); those too close to
// call go on a list.
__global__ void k_plan_again(const saber_region* __restrict__ reg, const DevPlan* __restrict__ plan,
                             const int32_t* __restrict__ sc, uint32_t n, const uint64_t* __restrict__ qoffs,
                             const uint64_t* __restrict__ soffs, const int64_t* __restrict__ region_floor, PlanParams P,
                             int32_t* __restrict__ score, uint8_t* __restrict__ again, uint32_t* __restrict__ ties,
                             uint32_t* __restrict__ nties) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t s = sc[i];
        score[i] = s;
        bool ag = false;
        if (plan[i].kind == 1) {
            const saber_region r = reg[i];
            bool tie = false;
            if (P.database_model) {
                ag = (double)s >= P.prefilter_frac * (double)region_floor[r.query];
            } else {
                // reaches the threshold of a bound of 1, or of the search space's
                const double wide = kTie * fabs(P.prefilter_frac) * (1.0 + 1.0 / P.lambda);
                auto reaches = [&](double f) {
                    if (P.even) f -= 1.0;
                    const double thr = P.prefilter_frac * f;
                    tie |= !(fabs((double)s - thr) > kTie * (fabs(thr) + 1.0) + wide);
                    return (double)s >= thr;
                };
                if (P.region_evalue > 0.0 && isfinite(P.region_evalue)) {
                    const int64_t qlen = (int64_t)(qoffs[r.query + 1] - qoffs[r.query]);
                    const int64_t sl = (int64_t)(soffs[r.subject + 1] - soffs[r.subject]);
                    double eps;
                    const double v = pl_adjustment(P, qlen, sl, eps), whole = rint(v);
                    auto with = [&](double up) {
                        return reaches(fmax(1.0, log(P.k * pl_space(P, qlen, sl, up) / P.region_evalue) / P.lambda));
                    };
                    if (fabs(v - whole) > eps || whole < 0.0) {
                        ag = with(ceil(fmax(v, 0.0)));
                    } else {  // the host may round it up to either
                        ag = with(whole);
                        tie |= !isfinite(v) || with(whole + 1.0) != ag;
                    }
                } else {
                    ag = reaches(1.0);
                }
                if (tie) ties[atomicAdd(nties, 1u)] = i;
            }
        }
        again[i] = ag;
    }
}

// What the host needs to decide a tie, and its answers.
struct TieRec {
    uint32_t query, slen;
    int32_t score;
};
__global__ void k_plan_ties(const saber_region* __restrict__ reg, const int32_t* __restrict__ score,
                            const uint64_t* __restrict__ soffs, const uint32_t* __restrict__ ties, uint32_t n,
                            TieRec* __restrict__ out) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const saber_region r = reg[ties[t]];
        out[t] = {r.query, (uint32_t)(soffs[r.subject + 1] - soffs[r.subject]), score[ties[t]]};
    }
}
__global__ void k_plan_untie(const uint32_t* __restrict__ ties, uint32_t n, const uint8_t* __restrict__ answers,
                             uint8_t* __restrict__ again) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) again[ties[t]] = answers[t];
}

__global__ void k_plan_jobs2(const saber_region* __restrict__ reg, const DevPlan* __restrict__ plan,
                             const uint32_t* __restrict__ list, uint32_t n2, const uint64_t* __restrict__ soffs,
                             saber_band_job* __restrict__ jobs) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x) {
        const uint32_t i = list[t];
        const saber_region r = reg[i];
        const DevPlan p = plan[i];
        jobs[t] = pl_job(r.query, r.subject, soffs[r.subject], p.lo, p.hi, p.blo, p.bhi);
    }
}

__global__ void k_plan_put(const uint32_t* __restrict__ list, uint32_t n2, const int32_t* __restrict__ sc,
                           int32_t* __restrict__ score) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x) score[list[t]] = sc[t];
}

// The regions that finish may report, with a margin on its f64 conditions.
__global__ void k_plan_keep(const saber_region* __restrict__ reg, const int32_t* __restrict__ score, uint32_t n,
                            const uint64_t* __restrict__ qoffs, const uint64_t* __restrict__ soffs,
                            const int64_t* __restrict__ floor, PlanParams P, uint8_t* __restrict__ keep) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t s = score[i];
        const saber_region r = reg[i];
        bool k;
        if (P.database_model) {
            k = (int64_t)s >= floor[r.query];
        } else {
            k = s > 0;
            const double adj = (double)(P.even && (s & 1) ? s - 1 : s);
            if (k && P.has_bits) {
                const double bits = (P.lambda * adj - P.log_k) / 0.69314718055994530942;
                k = !(bits < P.min_bitscore - kCutMargin * (fabs(P.min_bitscore) + 1.0));
            }
            if (k && isfinite(P.evalue_cut)) {
                const int64_t qlen = (int64_t)(qoffs[r.query + 1] - qoffs[r.query]);
                const int64_t sl = (int64_t)(soffs[r.subject + 1] - soffs[r.subject]);
                double eps;
                const double up = ceil(fmax(pl_adjustment(P, qlen, sl, eps), 0.0)) + 1.0;  // (the host's, or one more)
                k = !(P.k * pl_space(P, qlen, sl, up) * exp(-P.lambda * adj) > P.evalue_cut * (1.0 + kCutMargin));
            }
        }
        keep[i] = k;
    }
}

__global__ void k_plan_gather(const saber_region* __restrict__ reg, const uint32_t* __restrict__ src,
                              const DevPlan* __restrict__ plan, const int32_t* __restrict__ score,
                              const uint64_t* __restrict__ soffs, const uint32_t* __restrict__ list, uint32_t n,
                              KeptRegion* __restrict__ out) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t i = list[t];
        const saber_region r = reg[i];
        const DevPlan p = plan[i];
        KeptRegion o;
        o.query = r.query;
        o.subject = r.subject;
        o.d_min = r.d_min;
        o.d_max = r.d_max;
        o.best = r.best;
        o.score = score[i];
        o.src = src[i];
        o.sbase = soffs[r.subject];
        o.slen = (uint32_t)(soffs[r.subject + 1] - o.sbase);
        o.lo = p.lo;
        o.hi = p.hi;
        o.blo = p.blo;
        o.bhi = p.bhi;
        o.band = (uint32_t)p.band;
        o.pad_ = 0;
        out[t] = o;
    }
}

// Plans and scores the regions of the handle's last scan (sk, on the device).
int plan_and_score(saber_gpu* h, const RegionSink& sk, const PlanParams& P, const int64_t* floors,
                   const int64_t* region_floors, const PlanTie& tie, PlanResult& out) {
    out = PlanResult{};
    if (!sk.n) return SABER_OK;
    for (cudaEvent_t& e : h->pl_ev)
        if (!e) CU(h, cudaEventCreate(&e));
    const Dataset& ds = h->main;
    const QuerySet& qs = ds.qs;
    cudaStream_t s = h->stream;
    const uint32_t n = (uint32_t)sk.n;
    const saber_region* reg = sk.d_regs;
    const uint64_t* qoffs = qs.offsets.as<uint64_t>();
    const uint64_t* soffs = ds.soff.as<uint64_t>();
    const unsigned grid = nblocks(n, 256, h->sm_count * 32);
    CUALLOC(h, h->pl_key, (uint64_t)n * 8);
    CUALLOC(h, h->pl_keyo, (uint64_t)n * 8);
    CUALLOC(h, h->pl_idx, (uint64_t)n * 4);
    CUALLOC(h, h->pl_by, (uint64_t)n * 4);
    CUALLOC(h, h->pl_flag, (uint64_t)n + 8);
    CUALLOC(h, h->pl_list, (uint64_t)n * 4 + 8);
    CUALLOC(h, h->pl_span, (uint64_t)n * sizeof(int2));
    CUALLOC(h, h->pl_plan, (uint64_t)n * sizeof(DevPlan));
    CUALLOC(h, h->pl_score, (uint64_t)n * 4);
    CUALLOC(h, h->pl_floor, std::max<uint64_t>(qs.nq, 1) * 16);
    CUALLOC(h, h->pl_ctr, 64);
    uint32_t* ctr = h->pl_ctr.as<uint32_t>();  // 0 selected, 1 ties, words 2..3 banded regions
    CU(h, cudaMemsetAsync(ctr, 0, 64, s));
    int64_t* d_floor = h->pl_floor.as<int64_t>();
    int64_t* d_rfloor = d_floor + qs.nq;
    CU(h, cudaMemcpyAsync(d_floor, floors, (uint64_t)qs.nq * 8, cudaMemcpyHostToDevice, s));
    CU(h, cudaMemcpyAsync(d_rfloor, region_floors, (uint64_t)qs.nq * 8, cudaMemcpyHostToDevice, s));
    auto bits_for = [](uint64_t v) {
        int b = 1;
        while (b < 64 && (v >> b)) b++;
        return b;
    };
    const int bs = bits_for(ds.nsub ? ds.nsub - 1 : 0), bq = bits_for(qs.nq ? qs.nq - 1 : 0);
    unsigned long long *key = h->pl_key.as<unsigned long long>(), *keyo = h->pl_keyo.as<unsigned long long>();
    uint32_t *idx = h->pl_idx.as<uint32_t>(), *by = h->pl_by.as<uint32_t>(), *list = h->pl_list.as<uint32_t>();
    uint8_t* flag = h->pl_flag.as<uint8_t>();
    DevPlan* plan = h->pl_plan.as<DevPlan>();
    int32_t* score = h->pl_score.as<int32_t>();
    const thrust::counting_iterator<uint32_t> iota(0);
    size_t t1 = 0, t2 = 0;
    CU(h, cub::DeviceRadixSort::SortPairs(nullptr, t1, key, keyo, idx, by, (int)n, 0, bs + bq, s));
    CU(h, cub::DeviceSelect::Flagged(nullptr, t2, iota, flag, list, ctr, (int)n, s));
    CUALLOC(h, h->pl_tmp, std::max(t1, t2));  // (its own: scoring uses cub_tmp in captured graphs)
    auto select = [&]() -> int {
        size_t tb = h->pl_tmp.cap;
        CU(h, cub::DeviceSelect::Flagged(h->pl_tmp.p, tb, iota, flag, list, ctr, (int)n, s));
        return SABER_OK;
    };
    // spans of the pairs
    CU(h, cudaEventRecord(h->pl_ev[0], s));
    k_plan_keys<<<grid, 256, 0, s>>>(reg, n, bs, key, idx);
    size_t tb = h->pl_tmp.cap;
    CU(h, cub::DeviceRadixSort::SortPairs(h->pl_tmp.p, tb, key, keyo, idx, by, (int)n, 0, bs + bq, s));
    k_plan_flags<<<grid, 256, 0, s>>>(keyo, n, flag);
    int rc = select();
    if (rc != SABER_OK) return rc;
    k_plan_spans<<<nblocks(n, 128, h->sm_count * 32), 128, 0, s>>>(reg, by, list, ctr, n, P.hsp_threshold,
                                                                   h->pl_span.as<int2>());
    CU(h, cudaEventRecord(h->pl_ev[1], s));
    // stage 1
    rc = reserve_resident_jobs(h, n);
    if (rc != SABER_OK) return rc;
    k_plan_jobs<<<grid, 256, 0, s>>>(reg, h->pl_span.as<int2>(), n, qoffs, soffs, P, plan,
                                     h->jobs_dev.as<saber_band_job>(), reinterpret_cast<unsigned long long*>(ctr + 2));
    CU(h, cudaGetLastError());
    CU(h, cudaEventRecord(h->pl_ev[2], s));
    const double w0 = wall_ms();
    rc = score_resident_jobs(h, n, &out.stage1);
    if (rc != SABER_OK) return rc;
    const double w1 = wall_ms();
    float ms[2] = {0.f, 0.f};
    for (int i = 0; i < 2; i++) CU(h, cudaEventElapsedTime(&ms[i], h->pl_ev[i], h->pl_ev[i + 1]));
    out.spans_ms = ms[0];
    out.jobs_ms = ms[1];
    out.calls_ms = std::max(0.0, w1 - w0 - ms[0] - ms[1]);  // (the call's first wait is for the plans)
    // stage 2
    uint32_t* ties = by;  // (the group order is done with)
    k_plan_again<<<grid, 256, 0, s>>>(reg, plan, h->scores_dev.as<int32_t>(), n, qoffs, soffs, d_rfloor, P, score, flag,
                                      ties, ctr + 1);
    CU(h, cudaGetLastError());
    rc = select();
    if (rc != SABER_OK) return rc;
    uint32_t hc[4];
    CU(h, cudaMemcpyAsync(hc, ctr, 16, cudaMemcpyDeviceToHost, s));
    CU(h, cudaStreamSynchronize(s));
    out.banded = ((uint64_t)hc[3] << 32) | hc[2];
    if (hc[1]) {
        // decisions too close for the device: the host's libm decides
        const uint32_t nt = hc[1];
        CUALLOC(h, h->pl_ties, (uint64_t)nt * (sizeof(TieRec) + 1));
        TieRec* d_rec = h->pl_ties.as<TieRec>();
        uint8_t* d_answer = reinterpret_cast<uint8_t*>(d_rec + nt);
        std::vector<TieRec> rec(nt);
        std::vector<uint8_t> answer(nt);
        k_plan_ties<<<nblocks(nt, 256, h->sm_count * 32), 256, 0, s>>>(reg, score, soffs, ties, nt, d_rec);
        CU(h, cudaGetLastError());
        CU(h, cudaMemcpyAsync(rec.data(), d_rec, nt * sizeof(TieRec), cudaMemcpyDeviceToHost, s));
        CU(h, cudaStreamSynchronize(s));
        for (uint32_t t = 0; t < nt; t++) answer[t] = tie(rec[t].query, (int64_t)rec[t].slen, rec[t].score) ? 1 : 0;
        CU(h, cudaMemcpyAsync(d_answer, answer.data(), nt, cudaMemcpyHostToDevice, s));
        k_plan_untie<<<nblocks(nt, 256, h->sm_count * 32), 256, 0, s>>>(ties, nt, d_answer, flag);
        CU(h, cudaGetLastError());
        CU(h, cudaStreamSynchronize(s));  // (answer is this block's)
        rc = select();
        if (rc != SABER_OK) return rc;
        CU(h, cudaMemcpyAsync(hc, ctr, 4, cudaMemcpyDeviceToHost, s));
        CU(h, cudaStreamSynchronize(s));
    }
    const uint32_t n2 = hc[0];
    out.n2 = n2;
    out.stage2_ms = wall_ms() - w1;
    if (n2) {
        k_plan_jobs2<<<nblocks(n2, 256, h->sm_count * 32), 256, 0, s>>>(reg, plan, list, n2, soffs,
                                                                        h->jobs_dev.as<saber_band_job>());
        CU(h, cudaGetLastError());
        const double w2 = wall_ms();
        out.stage2_ms = w2 - w1;
        rc = score_resident_jobs(h, n2, &out.stage2);
        if (rc != SABER_OK) return rc;
        out.calls_ms += wall_ms() - w2;
        k_plan_put<<<nblocks(n2, 256, h->sm_count * 32), 256, 0, s>>>(list, n2, h->scores_dev.as<int32_t>(), score);
    }
    // what finish may report
    k_plan_keep<<<grid, 256, 0, s>>>(reg, score, n, qoffs, soffs, d_floor, P, flag);
    CU(h, cudaGetLastError());
    rc = select();
    if (rc != SABER_OK) return rc;
    CU(h, cudaMemcpyAsync(hc, ctr, 4, cudaMemcpyDeviceToHost, s));
    CU(h, cudaStreamSynchronize(s));
    out.n = hc[0];
    if (out.n) {
        CUALLOC(h, h->pl_kept, out.n * sizeof(KeptRegion));
        CUALLOC(h, h->pin_kept, out.n * sizeof(KeptRegion));
        k_plan_gather<<<nblocks(out.n, 256, h->sm_count * 32), 256, 0, s>>>(reg, sk.d_src, plan, score, soffs, list,
                                                                            (uint32_t)out.n, h->pl_kept.as<KeptRegion>());
        CU(h, cudaGetLastError());
        CU(h, cudaMemcpyAsync(h->pin_kept.p, h->pl_kept.p, out.n * sizeof(KeptRegion), cudaMemcpyDeviceToHost, s));
        CU(h, cudaStreamSynchronize(s));
        out.kept = h->pin_kept.as<KeptRegion>();
    }
    return SABER_OK;
}

}  // namespace saber
