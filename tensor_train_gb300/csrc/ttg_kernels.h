// Host-side launchers of the sweep, apply, eval and inner kernels.
#pragma once

#include <string>

#include <cuda_runtime.h>

#include "../../include/ttg.h"
#include "ttg_job.h"

namespace ttg
{

// ctas_per_sm: 1-2 (128 registers), 3 (85) or 4 (64): the instantiation.
void launch_round(const RoundJob& job, int grid, int ctas_per_sm, cudaStream_t stream);
// Whole-GPU rounding (cooperative launch, grid <= the value from setup).
cudaError_t launch_wide_round(const WideJob& job, int grid, cudaStream_t stream);
// Opt-in to the dynamic shared memory and the co-resident grid size.
cudaError_t wide_round_setup(int smem_doubles, int* max_grid);
void launch_apply_core(const double* A, const double* X, double* Y, int r, int m, int p, int rp,
                       int s, int nout, int sp, cudaStream_t stream);
// <a, b> of two TTs in `ar` into *out (cooperative).  scratch: z.scratch()
// doubles; bar: the launch's barrier word, whose err the caller reads.
struct InnerSizes;  // ttg_inner.h
cudaError_t launch_inner(const double* ar, const CoreSlot* SA, const CoreSlot* SB, int d,
                         const InnerSizes& z, double* scratch, GridBar* bar, double* out,
                         cudaStream_t stream);
cudaError_t round_smem_optin(int smem_doubles);
void launch_fp64_peak(double* out, int iters, int grid, int block, cudaStream_t stream);
// tcgen05 split-BF16 GEMM (ttg_tc_gemm.cu): C = A B (+ bias) (relu) (+ C),
// A taken as max(A, 0) with relu_a.  ws: a workspace of tc_gemm_ws_bytes kept
// by the caller (used in stream order), or null to allocate one for the call.
cudaError_t tc_gemm_f32(cudaStream_t st, int M, int N, int K, const float* A, int64_t a_rs,
                        int64_t a_cs, const float* B, int64_t b_rs, int64_t b_cs, float* C,
                        int64_t ldc, const float* bias, bool relu, bool accumulate, int splits,
                        bool relu_a = false, void* ws = nullptr);
size_t tc_gemm_ws_bytes(int M, int N, int K, int splits);
// Reads and clears the tensor-core GEMM timeout flag (synchronises st).
bool tc_gemm_timed_out(cudaStream_t st);
// ttg_eval_batch of M multi-indices that are part of a call with M_all: cut as
// for M_all, so that a split call's values do not depend on the split.
int32_t eval_batch_part(const ttg_tensor* a, const int32_t* idx, int32_t M, int32_t M_all,
                        double* out);
// Sets the message returned by ttg_last_error() on this thread.
void set_last_error(const std::string& msg);

}  // namespace ttg
