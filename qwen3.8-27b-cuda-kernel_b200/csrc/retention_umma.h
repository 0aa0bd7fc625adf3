// Shared between the translation units of retention (retention.cu, retention_umma.cu).
#pragma once

#include "host_util.h"

namespace q38 {

// Prefill with heads of 128 x 128 on the 5th-generation tensor cores: whether call and scratch allow it, and the launches.
bool retention_umma_fits(const q38_retention_params& p, const q38_batch_desc& b, const q38_recurrent_state_desc& st);
int retention_umma(const q38_retention_params& p, const q38_batch_desc& b, const q38_recurrent_state_desc& st, cudaStream_t s);

}  // namespace q38
