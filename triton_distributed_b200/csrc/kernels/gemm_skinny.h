// Few-row GEMMs: plan and launch, used by the dispatch in gemm_sm100.cu and gemm_fp8_sm100.cu.
#pragma once
#include "../include/tdist.h"

namespace tdist_host {

struct SkinnyPlan {
    int tok, m_tiles, n_tiles, split, stages, grid;
};

// True when the few-row kernel is expected to finish a plain product before `other_s` seconds (the estimate for the
// large-tile kernel); fills the plan. Looks at sizes only.
bool skinny_plan(int m, int n, int k, double other_s, SkinnyPlan* plan);
int skinny_run(const TdistGemmArgs* a, const SkinnyPlan& plan);

// The same for the block-scaled fp8 product (gemm_fp8_skinny_sm100.cu).
bool fp8_skinny_plan(int m, int n, int k, double other_s, SkinnyPlan* plan);
int fp8_skinny_run(const TdistGemmFp8Args* a, const SkinnyPlan& plan);

}  // namespace tdist_host
