// LDPCA rate-adaptive decoding on the device: the whole request ladder (start
// code from the conditional-entropy bound, syndrome of each ladder code from the
// accumulated syndrome, sum-product belief propagation with the parity early
// stop, CRC-8 acceptance, and the GF(2) inverse at full rate) with no host round
// trip between requests.
//
// Reference: DvcDec/src/LdpcaDecoder.cpp LdpcaDecoder (:646-771),
// beliefPropagation (:462-580), ComputeCE (:127-143), invH_mul (:624-643).
// The per-edge arithmetic, the order of every float sum (row sums in edge
// order, column sums in edge order, the entropy sum in block order) and the
// library functions (logf, tanhf via exact_libm) follow the reference exactly,
// so decoded bits, accepted codes and rates are identical to it.
//
// Two launch forms share one kernel:
//  * direct (K = 1, no scratch): one thread block per codeword walks the ladder
//    code by code, exactly as the reference does;
//  * speculative (K >= 1, scratch): K blocks per codeword try the ladder codes
//    start+k, start+k+K, ... concurrently.  A code is accepted by the reference
//    iff BP converges and the CRC matches and no lower code was accepted, i.e.
//    the accepted code is the lowest code that succeeds; blocks publish
//    successes with atomicMin, stop at (or abandon) codes above the best success
//    so far, and the last of the K blocks to finish (a counter with fences)
//    picks the lowest success (or the full-rate inverse when none), writes the
//    outputs and resets the codeword's scratch for the next launch, so results
//    are identical to the sequential ladder while idle SMs shorten it, with one
//    launch per bitplane step.
//
// The per-code BP, the syndrome, the inverse and the shared-memory layout are
// in ldpca_bp.cuh.
#include <cuda_runtime.h>

#include <stdlib.h>

#include <algorithm>

#include "dvc_common.cuh"
#include "dvc_types.h"
#include "kernels.h"
#include "ldpca_bp.cuh"

namespace dvc {

// One thread block of NT threads per (codeword, speculative slot), or a cluster
// of C of them, each thread holding MAXC = ceil(n / (C * NT)) columns, MINB
// blocks per SM.  Alone NT = 1024 for both lengths (CIF: one block per SM, 105
// KB of shared memory; QCIF: 27 KB); QCIF codewords can also run with 256 or
// 512 threads, four or two blocks per SM (the autotuner measures which is faster).
// ANY: a codeword of any length up to NT * MAXC; without it of a length that
// needs all MAXC rounds, which spares the edge pass a bound.
template <int NT, int MAXC, int MINB, int C, bool ANY>
__global__ void __launch_bounds__(NT, MINB)
    ldpca_ladder_kernel(LadderDev L, const LdpcaJob *__restrict__ jobs, XlmDev xt, int max_iter, int K,
                        LdpcaSpec sp) {
  extern __shared__ __align__(16) uint8_t smem[];
  // codeword j and its speculative slot kk: the first slots of all codewords
  // come first, so that blocks waiting for an SM are those of later codes
  const int unit = blockIdx.x / C, nj = gridDim.x / (C * K);
  const int kk = unit / nj, j = unit - kk * nj, slot = j * K + kk;
  const LdpcaJob J = jobs[j];
  if (!J.active) return;
  const bool spec = sp.best != nullptr;
  using G = LdGroup<NT, true, C, ANY>;
  const G g{(int)threadIdx.x, 0, C > 1 ? (int)blockIdx.x - unit * C : 0};
  const int n = L.n, tid = threadIdx.x;
  const bool lead = tid == 0 && g.rank == 0;
  const LdSmem S = ld_carve(smem, L);
  __shared__ uint32_t s_ured[NT / 32];
  __shared__ LdCtl s_ctl;
  __shared__ int s_word[4];  // broadcast words: late, start code, then stop flags in turn
  __shared__ uint4 s_pdesc[XL_PHI_MAX_SEGS];
  const XlSmall xs = xl_small_global(xt);
  xl_phi_stage(xt, s_pdesc);
  if constexpr (C > 1) g.sync_all();  // every block of the cluster has started
  const int last = L.num_codes - 1;
  int total_iters = 0, accepted = last, start = 0;
  // a slot that starts after its codeword has been decoded by a lower code
  // than its own has nothing to do
  bool late = false;
  // the slot that reports the bound: an early one, which has an SM from the
  // start even when there are more slots than SMs (the last one held up every
  // bitplane step of a lone CIF frame by 13 us)
  const int reporter = min(K - 1, 3);
  if (spec && kk > 0 && kk != reporter) {
    int l = 0;
    if (lead) {
      const int best = *(volatile int *)(sp.best + j);
      __threadfence();
      l = best != LDPCA_NONE && *(volatile int *)(sp.start + j) + kk > best;
    }
    late = g.bcast(l, &s_word[0]) != 0;
    if (late) start = *(volatile int *)(sp.start + j);
  }
  if (!late) {

  // accumulated syndrome bits (ByteToBit, LdpcaDecoder.cpp:81-107), log LR and
  // the entropy terms (ComputeCE), the bound as a sequential sum in block order
  float llr[MAXC], part = 0.0f;
  ld_llr(g, n, J.lr, xt, xs, llr, J.use_given_entropy ? nullptr : S.msg, (J.llr_out && kk == 0) ? J.llr_out : nullptr,
         J.llr_in, J.term_in, &part);
  ld_stage_acc(g, J.acc, n, S.accs);
  if (J.use_given_entropy) g.sync_all();  // the staged syndrome; otherwise ld_start_near's barriers
  // The bound itself is only needed where it is reported and when the parallel
  // sum leaves the start code open.
  start = J.use_given_entropy ? ld_start_code(L, J.given_entropy) : ld_start_near(g, L, part, s_ured, &s_ctl);
  if (J.use_given_entropy) {
    if (lead && kk == reporter && J.entropy) *J.entropy = J.given_entropy;
  } else if (start < 0 || kk == reporter) {
    g.sync_all();
    int exact = start;
    if (lead) {
      const float h = ld_entropy_sum(S.msg, n);
      if (exact < 0) exact = ld_start_code(L, h);
      if (J.entropy && kk == reporter) *J.entropy = h;
    }
    start = g.bcast(exact, &s_word[1]);
  }
  if (spec && lead) *(volatile int *)(sp.start + j) = start;  // the same in every slot
  volatile int *bestp = spec ? sp.best + j : nullptr;

  int turn = 0;
  for (int code = start + kk; code < last; code += K) {
    if (spec) {
      if (g.bcast(lead && *bestp < code, &s_word[2 + turn])) break;
      turn ^= 1;
    }
    int it = 0;
    uint32_t dm = 0;
    const int ok = ld_try_code(g, L, code, llr, J.crc, xt, s_pdesc, max_iter, bestp, S, s_ured, &s_ctl, it, dm);
    total_iters += it;
    if (spec && sp.code_iters && lead) sp.code_iters[j * LDPCA_TRIED + code - start] = it;
    if (ok) {
      accepted = code;
      if (spec) {
        uint8_t *dec = sp.slot_dec + (size_t)slot * n;
        for (int c = 0; c < MAXC; c++) {
          const int k = g.col(n, c);
          if (k < n) dec[k] = (uint8_t)((dm >> c) & 1u);
        }
        __threadfence();
        g.sync_all();
        if (lead) {
          sp.slot_code[slot] = code;
          __threadfence();
          atomicMin(sp.best + j, code);
        }
      }
      break;
    }
  }
  }
  if (spec) {
    // the last of the codeword's K slots to finish writes its result (in a
    // cluster its first block does): the lowest successful code (or the
    // full-rate code when no code below it succeeded), then puts the
    // codeword's scratch back to its initial state
    // for the next launch (no memset between the steps of a batch)
    __shared__ int s_last, s_slot, s_iters, s_acc;
    g.sync_all();  // nothing in a block's shared memory is read by another one after this
    if (C > 1 && g.rank != 0) return;
    if (tid == 0) {
      atomicAdd(sp.iters + j, total_iters);
      __threadfence();
      s_last = atomicAdd(sp.done + j, 1) == K - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (tid == 0) {
      const int best = __ldcg(sp.best + j);
      int acc = last, from = -1;
      if (best != LDPCA_NONE && best < last)
        for (int k = 0; k < K; k++)
          if (__ldcg(sp.slot_code + j * K + k) == best) {
            from = k;
            acc = best;
          }
      s_acc = acc;
      s_slot = from;
      // the BP iterations of the sequential ladder (every code up to the
      // accepted one ran to its end), or those of every code tried
      int iters = 0;
      if (sp.code_iters)
        for (int c = start; c <= min(acc, last - 1); c++) iters += __ldcg(sp.code_iters + j * LDPCA_TRIED + c - start);
      else
        iters = __ldcg(sp.iters + j);
      s_iters = iters;
    }
    __syncthreads();
    accepted = s_acc;
    if (s_slot >= 0) {
      const uint8_t *src = sp.slot_dec + (size_t)(j * K + s_slot) * n;
      for (int k = tid; k < n; k += NT) S.dec[k] = __ldcg(src + k);
    }
    total_iters = s_iters;
    for (int k = tid; k < K; k += NT) sp.slot_code[j * K + k] = -1;
    if (tid == 0) {
      sp.best[j] = LDPCA_NONE;
      sp.iters[j] = 0;
      sp.done[j] = 0;
    }
  }
  __syncthreads();
  const LdGroup<NT, true> b{tid, 0, 0};
  if (accepted == last) ld_full_rate(b, L, S);
  if (tid == 0) {
    J.result[0] = L.synd_len[accepted] + 8;
    J.result[1] = start;
    J.result[2] = accepted;
    J.result[3] = total_iters;
  }
  if (J.decoded)
    for (int k = tid; k < n; k += NT) J.decoded[k] = S.dec[k];
  if (J.recons_trans) ld_put_bitplane(b, J, S.dec, n);
}

// the L2 persisting window of the table reads (set when a context is created;
// process-wide like the launch shapes)
static cudaAccessPolicyWindow g_phi_window = {};

void set_phi_window(const void *base, size_t num_bytes, float hit_ratio) {
  g_phi_window = cudaAccessPolicyWindow{};
  if (!base || num_bytes == 0) return;
  g_phi_window.base_ptr = const_cast<void *>(base);
  g_phi_window.num_bytes = num_bytes;
  g_phi_window.hitRatio = hit_ratio;
  g_phi_window.hitProp = cudaAccessPropertyPersisting;
  g_phi_window.missProp = cudaAccessPropertyStreaming;
}

// the window as a launch attribute; returns the number of attributes (0 or 1)
unsigned phi_window_attr(cudaLaunchAttribute &a) {
  if (g_phi_window.num_bytes == 0) return 0;
  a.id = cudaLaunchAttributeAccessPolicyWindow;
  a.val.accessPolicyWindow = g_phi_window;
  return 1;
}

template <int NT, int MAXC, int MINB, int C = 1, bool ANY = false>
static cudaError_t launch_nt(const LadderDev &L, const LdpcaJob *jobs, int num_jobs, const XlmDev &xt, int max_iter,
                             int K, const LdpcaSpec &sp, cudaStream_t stream) {
  const int rounds = LDPCA_COLS(L.n, NT * C);
  if (L.n > LDPCA_MAX_N || (ANY ? rounds > MAXC : rounds != MAXC)) return cudaErrorInvalidValue;
  auto kernel = ldpca_ladder_kernel<NT, MAXC, MINB, C, ANY>;
  const size_t smem = ldpca_smem_bytes(L);
  // the rest of the SM's 256 KB is L1 for the phi records, which BP iterations re-read
  static SmemLimit limit;
  const cudaError_t e = limit.raise(kernel, smem, MINB);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_jobs * K * C);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = phi_window_attr(attr[0]);
  if (C > 1) {
    cudaLaunchAttribute &a = attr[cfg.numAttrs++];
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = C;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, L, jobs, xt, max_iter, K, sp);
}

// threads per codeword block: CIF 1024 (or 512), QCIF 1024 (or 256, 512)
static int g_ldpca_threads = 1024, g_ldpca_threads_qcif = 1024;

void set_ldpca_threads(int nt, int nt_qcif) {
  g_ldpca_threads = (nt == 512) ? 512 : 1024;
  g_ldpca_threads_qcif = (nt_qcif == 256 || nt_qcif == 512) ? nt_qcif : 1024;
}

static cudaError_t launch_shape(const LadderDev &L, const LdpcaJob *jobs_dev, int num_jobs, const XlmDev &xt,
                                int max_iter, int K, const LdpcaSpec &sp, cudaStream_t stream) {
  if (L.n == 1584) {
    if (g_ldpca_threads_qcif == 1024) return launch_nt<1024, 2, 1>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
    if (g_ldpca_threads_qcif == 512) return launch_nt<512, 4, 2>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
    return launch_nt<256, 7, 4>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  }
  if (L.n != LDPCA_MAX_N) return launch_nt<1024, 7, 1, 1, true>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  if (g_ldpca_threads == 512) return launch_nt<512, 13, 1>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  return launch_nt<1024, 7, 1>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
}

cudaError_t launch_ldpca(const LadderDev &L, const LdpcaJob *jobs_dev, int num_jobs, const XlmDev &xt, int max_iter,
                         cudaStream_t stream) {
  if (num_jobs <= 0) return cudaSuccess;
  LdpcaSpec none{};
  return launch_shape(L, jobs_dev, num_jobs, xt, max_iter, 1, none, stream);
}

// Slots beyond those the SMs hold at once cost little (they start in code order
// and find their codeword decoded), and hard codewords need many: four times
// the SMs, at least 4 and at most 32 slots a codeword.  Measured with once,
// twice and four times the SMs: three GOP-8 QCIF streams 147, 114, 106 ms, four
// GOP-4 CIF streams 246, 196, 183 ms, 54 mixed requests 57, 48, 48 ms; 64 slots
// instead of 32 slow a lone frame by 0.1-0.3 ms.  When fewer codewords are
// active than the SMs could serve, a slot is a cluster of C blocks: a BP
// iteration on 1, 2, 4 and 8 blocks takes 46, 35, 21 and 13 K cycles at CIF and
// 13, 11, 8.3 and 7.8 K at QCIF (a remote store per edge, and the latency of two
// table gathers, do not shrink with C).  So CIF keeps four slots per codeword
// resident (a lone CIF frame 11.5 -> 6.5 ms at C = 8, four frames 24 -> 12 ms,
// eleven at QIndex 8 80 -> 73 ms at C = 2; six or three slots instead of four:
// four frames 14.6 or 12.3 ms), and QCIF, which gains less, sixteen (a lone
// frame 3.45 -> 3.04 ms at C = 4; with eight, the three QCIF streams lose 5%).
// A codeword of another length (a ladder file may hold any up to LDPCA_MAX_N)
// keeps one block per slot: the cluster shapes are cut for these two.
// DVC_LDPCA_SPEC_FLOOR replaces the least number of slots (the autotuner's
// setting), DVC_LDPCA_SPEC fixes it outright.
void ldpca_spec_shape(int n, int active, int sms, int &K, int &C) {
  const int N = std::max(1, active);
  const bool small = n < LDPCA_MAX_N;
  const int resident = small ? 16 : 4;
  C = n == 1584 ? 4 : n == LDPCA_MAX_N ? 8 : 1;
  while (C > 1 && N * C * resident > sms) C /= 2;
  int least = 4;
  if (const char *e = getenv("DVC_LDPCA_SPEC_FLOOR")) least = std::max(1, std::min(32, atoi(e)));
  K = std::max(least, 4 * sms / (N * C));
  if (const char *e = getenv("DVC_LDPCA_SPEC")) K = atoi(e);
  K = std::max(1, std::min(32, K));
}

size_t ldpca_spec_scratch_bytes(int n, int num_jobs, int K) {
  return (size_t)num_jobs * 16 + (size_t)num_jobs * K * 4 + (size_t)num_jobs * K * n +
         (size_t)num_jobs * LDPCA_TRIED * 4 + 64;
}

LdpcaSpec ldpca_spec_carve(void *base, int num_jobs, int K, bool code_iters) {
  LdpcaSpec sp;
  uint8_t *p = (uint8_t *)base;
  sp.best = (int *)p;
  p += (size_t)num_jobs * 4;
  sp.iters = (int *)p;
  p += (size_t)num_jobs * 4;
  sp.start = (int *)p;
  p += (size_t)num_jobs * 4;
  sp.done = (int *)p;
  p += (size_t)num_jobs * 4;
  sp.slot_code = (int *)p;
  p += (size_t)num_jobs * K * 4;
  if (code_iters) sp.code_iters = (int *)p;
  p += (size_t)num_jobs * LDPCA_TRIED * 4;
  sp.slot_dec = p;
  return sp;
}

cudaError_t ldpca_spec_reset(const LdpcaSpec &sp, int num_jobs, int K, cudaStream_t stream) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(sp.best, 0x7f, (size_t)num_jobs * 4, stream)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(sp.iters, 0, (size_t)num_jobs * 4, stream)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(sp.done, 0, (size_t)num_jobs * 4, stream)) != cudaSuccess) return e;
  return cudaMemsetAsync(sp.slot_code, 0xff, (size_t)num_jobs * K * 4, stream);
}

cudaError_t launch_ldpca_spec(const LadderDev &L, const LdpcaJob *jobs_dev, int num_jobs, const XlmDev &xt,
                              int max_iter, int K, int C, const LdpcaSpec &sp, cudaStream_t stream) {
  if (num_jobs <= 0) return cudaSuccess;
  // threads per block: the columns of a block in whole rounds
  if (L.n == 1584 && C == 4) return launch_nt<416, 1, 1, 4>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  if (L.n == 1584 && C == 2) return launch_nt<800, 1, 1, 2>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  if (L.n == 6336 && C == 8) return launch_nt<800, 1, 1, 8>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  if (L.n == 6336 && C == 4) return launch_nt<800, 2, 1, 4>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  if (L.n == 6336 && C == 2) return launch_nt<800, 4, 1, 2>(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
  if (C != 1) return cudaErrorInvalidValue;
  return launch_shape(L, jobs_dev, num_jobs, xt, max_iter, K, sp, stream);
}

}  // namespace dvc
