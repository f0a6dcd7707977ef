// The scan's hand-off of candidate regions to the host batch engine (plain
// C++, shared by the CUDA translation units and engine.cpp).
#pragma once
#include <cstdint>
#include <functional>

#include "saber_gpu.h"

namespace saber {

// The batch engine's candidate regions, capped per query (and triaged): the
// kept regions in region order (grouped by query) with their positions in the
// capped list, in device memory owned by the handle (valid until its next
// scan).
struct RegionSink {
    float lambda = 0.f, logk = 0.f;  // for the triage features
    const saber_region* d_regs = nullptr;
    const uint32_t* d_src = nullptr;
    uint64_t n = 0;                  // kept regions
    uint64_t ncap = 0;               // regions after the per-query cap
    bool triaged = false;            // a model dropped regions
    bool collecting = false;         // feature rows were collected
    double triage_ms = 0;            // wall clock of the features, the network and its cut
};

// What planning and scoring the regions needs of the search's parameters and
// of the statistics (one query's numbers aside).
struct PlanParams {
    int64_t window_slack, score_band, prefilter_band;
    int32_t hsp_threshold;
    int32_t database_model, even, has_bits;
    double prefilter_frac, region_evalue, evalue_cut, min_bitscore;
    double lambda, k, log_k, adl, beta, num_seqs;
};

// A planned and scored region that may be reported.
struct KeptRegion {
    uint32_t query, subject;
    int32_t d_min, d_max, best, score;
    uint32_t src, slen;
    uint64_t sbase;
    int32_t lo, hi, blo, bhi;  // the plan: window, band
    uint32_t band;             // the plan is banded
    uint32_t pad_;
};
static_assert(sizeof(KeptRegion) == 64, "one record is 64 bytes");

// Whether a region (query, subject length, stage-1 score) goes on to the second
// stage: the host's answer where the device's f64 is too close to the threshold.
using PlanTie = std::function<bool(uint32_t, int64_t, int32_t)>;

struct PlanResult {
    const KeptRegion* kept = nullptr;  // pinned memory of the handle, valid until its next search
    uint64_t n = 0;
    uint64_t banded = 0;  // regions with a banded plan
    uint64_t n2 = 0;      // regions scored again
    saber_score_stats stage1{}, stage2{};
    double spans_ms = 0, jobs_ms = 0;    // device time: the pairs' spans; plans and first-stage jobs
    double calls_ms = 0, stage2_ms = 0;  // wall clock: the scoring calls; second-stage decisions and jobs
};

}  // namespace saber
