// The channel-last form of the Mamba1 scan (sscan_cl.cu), entered through qb_sscan_fwd.
#pragma once
#include "common.cuh"
namespace qb {
int run_sscan_channel_last(const qb_sscan_fwd_args& a, cudaStream_t st);
int64_t sscan_workspace_bytes(int batch, int dim);
}
