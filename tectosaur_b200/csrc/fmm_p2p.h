// P2P on a work plan (fmm_p2p.cu), as fmm.cu calls it.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace tct {

struct P2PCall {
    const double *qp, *qw, *params;  // host rule and elastic constants
    const void* obs_pts;
    const int32_t* obs_tris;         // tree order
    const void* src_pts;
    const int32_t* src_tris;         // tree order
    int64_t n_src;
    const int64_t* src_orig;         // input row of a tree-ordered source
    const void* in;
    const void* rec;                 // far_prep's records (other kernels than elasticRH3)
    void* W;                         // sums per tree-ordered obs triangle (out)
    unsigned char* ws;
};

bool p2p_is_rh(int kernel, int nq);
size_t p2p_workspace_bytes(int kernel, int prec, int nq, int64_t n_src,
                           const tct_fmm_p2p_plan& plan);
int p2p_planned(int kernel, int prec, int nq, const P2PCall& k, const tct_fmm_p2p_plan& plan,
                cudaStream_t st);

}  // namespace tct
