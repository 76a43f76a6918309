// First stage of a top-k search over many keys (tq_score_filter.cu), as the scoring path (tq_score_tc.cu) uses it.
#pragma once

#include "tq_common.cuh"

// One pass of at most 64 queries: where its lists, the gathered keys and the results of a round live (device pointers).
struct TqFilterPass {
    int nq, qpad;
    int cap;                     // entries per list
    int room;                    // keys the gathered arrays hold
    float beta_scale;
    unsigned char* fprep;        // tq_filter_prep_bytes
    float* thr;                  // [nq]
    unsigned int* cnt;           // [nq]
    unsigned int* rows;          // [nq][cap]
    unsigned int* offsets;       // [nq]
    unsigned int* bad;           // set: some list or the gathered arrays were too small, or a query is beyond the bound
    unsigned int* gathered;      // keys gathered
    unsigned int* expected;      // [kFilterRounds] keys the rounds will list, by the sample
    uint32_t *g_codes, *g_signs;
    float *g_norms, *g_rnorms;
    unsigned int* g_rows;
    float* scores;               // [nq][room]
    unsigned long long* best;    // [nq][topk]
};

size_t tq_filter_prep_bytes(int d, int qpad);
int tq_launch_filter_prep(const tq_plan* p, const unsigned char* prep, int qpad, int nq, float c_max, float beta_scale, unsigned char* out,
                          unsigned int* bad, cudaStream_t st);
// What the rounds multiply the sample by, so that the sample can tell how many keys each round will list.
constexpr int kFilterRounds = 16;
struct TqFilterRounds {
    int rounds;
    float keys[kFilterRounds];       // keys of round r over those of the sample
};
int tq_launch_sample_threshold(const TqFilterPass& f, const TqFilterRounds& rounds, const unsigned long long* cand, int64_t cap, int topk, cudaStream_t st);
int tq_launch_filter(const tq_plan* p, const TqFilterPass& f, const uint32_t* codes, const uint32_t* signs, const float* rnorms,
                     const float* norms, int64_t keys, int tile_stride, cudaStream_t st);
int tq_launch_filter_gather(const tq_plan* p, const TqFilterPass& f, const uint32_t* codes, const uint32_t* signs, const float* rnorms,
                            const float* norms, cudaStream_t st);
int tq_launch_filter_select(const TqFilterPass& f, int topk, int k2, bool final, bool keep_nan, cudaStream_t st);
