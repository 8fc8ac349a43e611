// One kind of the few-rows kernel: int8 weights, bf16 activations (a file of its own so that they compile side by side).
#include "qmm_rows.cuh"

template int qmm::rows::launch_rows_kernel<qmm::rows::kAff8, __nv_bfloat16>(const CUtensorMap&, const CUtensorMap&, qmm::rows::RowsParams&, qmm::rows::RowsPlan&,
                                                                    const qmm::rows::RowsShape&, bool, cudaStream_t);
