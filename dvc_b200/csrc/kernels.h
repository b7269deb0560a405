// Launch entry points of the decoder kernels (host side).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "dvc_types.h"
#include "libm_tables.h"

namespace dvc {

// A kernel's dynamic shared memory limit and preferred carveout, set per device
// and raised when a launch needs more than every one before it: what a ladder
// kernel needs depends on the ladder file of the context (the padding of its
// rows), and a process may hold contexts on several.
struct SmemLimit {
  std::mutex mu;
  std::atomic<size_t> most[64] = {};
  // for the current device; blocks: those of `smem` dynamic bytes, and 12 KB of
  // its own, that an SM is to hold (the carveout is the smallest split that
  // does, so that the rest is L1; percent of the 228 KB maximum, the driver
  // rounds up to a supported split)
  template <class Kernel>
  cudaError_t raise(Kernel kernel, size_t smem, int blocks) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::atomic<size_t> &m = most[dev & 63];
    if (smem <= m.load()) return cudaSuccess;
    std::lock_guard<std::mutex> lk(mu);
    if (smem <= m.load()) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const size_t need = (size_t)blocks * (smem + 12 * 1024);
    const int pct = (int)std::min<size_t>(100, (need * 100 + 228 * 1024 - 1) / (228 * 1024));
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
    if (e == cudaSuccess) m.store(smem);
    return e;
  }
};

// direct form: one block per codeword, no scratch
cudaError_t launch_ldpca(const LadderDev &L, const LdpcaJob *jobs_dev, int num_jobs, const XlmDev &xt,
                         int max_iter, cudaStream_t stream);
// speculative form: K slots per codeword, each a block or a cluster of C = 2, 4
// or 8 blocks, the last of them writes the result (with code_iters in the
// scratch, the BP iterations of the sequential ladder in it; else of every code tried);
// scratch from ldpca_spec_carve, put in its initial state once by
// ldpca_spec_reset (each launch leaves it so for the next)
// slots per codeword (K) and blocks per slot (C) for `active` codewords of n
// bits decoding at once on `sms` multiprocessors
void ldpca_spec_shape(int n, int active, int sms, int &K, int &C);
size_t ldpca_spec_scratch_bytes(int n, int num_jobs, int K);
LdpcaSpec ldpca_spec_carve(void *base, int num_jobs, int K, bool code_iters = false);
cudaError_t ldpca_spec_reset(const LdpcaSpec &sp, int num_jobs, int K, cudaStream_t stream);
cudaError_t launch_ldpca_spec(const LadderDev &L, const LdpcaJob *jobs_dev, int num_jobs, const XlmDev &xt,
                              int max_iter, int K, int C, const LdpcaSpec &sp, cudaStream_t stream);
// threads per codeword block of the ladder kernel: CIF 1024 or 512, QCIF 1024,
// 512 or 256 (other values select the defaults, 1024 for both)
void set_ldpca_threads(int nt, int nt_qcif);
// threads per updateSI tile (256 or 512) and per forward motion search block
// (128, 256 or 512); other values select 256
void set_me_shapes(int si_threads, int fme_threads);
// L2 persisting access window of the LDPCA kernels' table reads (num_bytes 0: none)
void set_phi_window(const void *base, size_t num_bytes, float hit_ratio);
// batched form: one persistent launch over codewords of both lengths
// (k_ldpca_batch.cu); state + slot bytes per codeword from ldpca_batch_state_bytes
size_t ldpca_batch_state_bytes(int count);
cudaError_t launch_ldpca_batch(LdpcaBatch A, int count, int grid, cudaStream_t stream);
// encoder: accumulated syndromes (n/8 bytes, MSB first) and CRC-8 of `count` source bitplanes
cudaError_t launch_ldpca_encode(const LadderDev &L, const uint8_t *bits_dev, int count, uint8_t *acc_dev,
                                uint8_t *crc_dev, cudaStream_t stream);

}  // namespace dvc
