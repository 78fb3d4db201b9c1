// The one-kernel accumulator encoder (ck_ldpc_encode.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ck {

// Encodes B frames (ck_ldpc_encode's accumulator form); *bad, where given, is
// set to 1 when an information byte is not 0 or 1.  *done is false, and
// nothing is launched, for codes whose information bits exceed a block's
// shared memory.
int encode_accumulate(const int8_t* info, int64_t B, int32_t k, int32_t m, int32_t n, const int32_t* row_ptr,
                      const int32_t* cols, int32_t g, int8_t* words, int32_t* bad, cudaStream_t stream, bool* done);

}  // namespace ck
