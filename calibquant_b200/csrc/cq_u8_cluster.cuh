// Interface between the uint8-format decode entry point (cq_calibquant.cu) and its single-launch path (cq_u8_cluster.cu).
#pragma once

#include "cq_common.cuh"

namespace cq {

// Requests whose scores fit the shared memory of a cluster, with 16-byte aligned full-precision rows.
bool u8_cluster_eligible(const cq_u8_decode_args* a);
int u8_cluster_run(const cq_u8_decode_args* a, void* status_word, cudaStream_t stream);

}  // namespace cq
