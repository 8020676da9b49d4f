// The FP64 row operator of a context (context_rows.cu).
#pragma once

#include "context_internal.cuh"
#include "kernels_rows.cuh"

namespace cfem {
namespace detail {

RowOp op_of(cfem_ctx *c, const RowsValues &V);

}  // namespace detail
}  // namespace cfem
