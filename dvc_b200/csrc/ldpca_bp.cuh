// Device building blocks of LDPCA rate-adaptive decoding, shared by the
// frame-batch ladder kernel (k_ldpca.cu) and the persistent work-queue kernel
// (k_ldpca_batch.cu).
//
// Reference: DvcDec/src/LdpcaDecoder.cpp LdpcaDecoder (:646-771),
// beliefPropagation (:462-580), ComputeCE (:127-143), invH_mul (:624-643),
// bitplane.cpp putBitplaneToCoeff (:4-22).  The per-edge arithmetic, the order
// of every float sum (row sums in edge order, column sums in edge order, the
// entropy sum in block order) and the library functions (logf, tanhf via
// exact_libm) follow the reference exactly.
//
// A codeword is decoded by a group of NT threads: a whole thread block, or one
// of several equal parts of a block, each synchronising on its own named
// barrier (bar.sync id, NT), so that a block of 1024 threads can work on one
// CIF codeword (n = 6336) or on four QCIF codewords (n = 1584) at once with the
// same shared memory.  Each thread keeps the log-LRs of its columns
// (k = t, t + NT, ...) in registers: MAXC = ceil(n / NT) of them.
//
// A codeword may also be shared by a cluster of C thread blocks (C > 1), each
// taking every C-th group of rows and a contiguous share of the columns; the
// edge messages live in the shared memory of the block that owns their row and
// are written there through distributed shared memory.
//
// One BP iteration is two passes with a barrier after each:
//   rows:  the sum of a row's magnitudes in edge order, its sign parity with
//          the syndrome bit (the sum's sign bit carries it), and whether the
//          row's check holds for the last hard decision;
//   edges: a column's thread forms its three incoming messages
//          phi(row sum - own magnitude), their total, the hard decision and
//          the three outgoing magnitudes phi(|total - incoming|), with nothing
//          stored in between.
// The message of an edge is one float: its magnitude (phi >= 0) with the sign
// of the message in the sign bit.  A check is tracked by a bit per row that
// starts as the syndrome bit and is flipped when a column's decision changes
// (few do after the first iterations), so no decision is stored per edge.
// What bounds it: each magnitude phi(y) = -logf(tanhf(y)) is one 16-byte record
// gathered from the packed table (dvc_common.cuh), two per edge and iteration,
// and an SM takes one random 32-byte sector per cycle from L2 (measured: 1.0
// cycle per gather for hot tables up to 64 MB and at least about 90 KB of L1,
// half that rate with a small L1): 38,016 cycles for a CIF codeword.  An
// iteration takes 46.9 K (41 K in the edge pass, 5.4 K in the row pass); three
// passes with separate sign and decision bytes took 65 K, this form with a
// 72 MB hot table (36 MB now) 50.7 K.  Two columns of a thread in flight at once
// change nothing at 1024 threads, three at 704 threads take 54 K.
// Rows are stored transposed in groups of 32 of similar degree (LadderDev), so
// the row pass reads without bank conflicts and spends its time on the sums.
//
// Shared memory per codeword (n bits, P = pos_max positions; CIF P = 19,072:
// 102 KB; QCIF 27 KB):
//   msg[P]    f32  edge messages
//   rowt      f32  row sums by slot, with the parity sign (after decoding: the
//                  decoded bits, one byte each)
//   hdr       uint4 per row group: its place, the syndrome bits of its rows,
//                  the rows whose check fails, its width
//   accs[n/8]      the packed accumulated syndrome, staged once per codeword
#pragma once
#include <cuda_runtime.h>

#include "dvc_common.cuh"
#include "dvc_types.h"

namespace dvc {

#define LDPCA_LOG2 (0.693147181f)  // LdpcaDecoder.cpp:18
#define LDPCA_NONE 0x7f7f7f7f      // "no success yet" (memset pattern 0x7f)

// rounds (columns per thread) of a group of nt threads on codewords of n bits
#define LDPCA_COLS(n, nt) (((n) + (nt) - 1) / (nt))

__host__ __device__ inline size_t ldpca_smem_bytes(const LadderDev &L) {
  size_t b = (size_t)L.pos_max * 4;        // msg
  b += (size_t)L.groups * 16;              // hdr
  b += (size_t)L.groups * 32 * 4;          // rowt (n words or more: the full-rate code has n rows)
  b += (size_t)L.n / 8;                    // accs
  return (b + 15) & ~(size_t)15;
}

// shared words a group coordinates through (one set per group)
struct LdCtl {
  uint32_t any[2];  // cluster form: a check failed (by iteration parity)
  uint32_t stop;    // a lower code of the codeword has succeeded
  uint32_t crc[8];  // cluster form: each block's part of the CRC
  int flag;         // free for the caller, and the CRC's verdict
};

// distributed shared memory: the address of this block's shared word in block
// `rank` of the cluster, and a store and an xor there
__device__ __forceinline__ uint32_t ld_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void ld_st_cluster(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void ld_xor_cluster(uint32_t addr, uint32_t v) {
  asm volatile("red.relaxed.cluster.shared::cluster.xor.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void ld_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// an edge word of the edge pass; volatile, so that it is not loaded before the
// row pass and waited for there
__device__ __forceinline__ uint32_t ld_edge(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// NT threads decoding one codeword (or, in a cluster of C blocks, NT threads of
// each block); `t` is the thread's index in its block's part.  BLOCK: the group
// is the whole thread block and synchronises with the block's barrier
// (__syncthreads); otherwise on the hardware barrier `bar` (1-15), which only
// its NT threads use.  ANY: codewords of any length, whose rounds may be fewer
// than the caller's loops; otherwise of one that fills them all.
template <int NT_, bool BLOCK, int C_ = 1, bool ANY_ = false>
struct LdGroup {
  static constexpr int NT = NT_, C = C_, STRIDE = NT_ * C_;
  static_assert(C_ == 1 || BLOCK, "a cluster group takes whole blocks");
  int t, bar, rank;
  // Columns of a thread, one per round.  When n is not a multiple of STRIDE
  // the first round is a partial one: its columns (the last of the codeword)
  // are spread over all warps, a few lanes of each, and the full rounds
  // follow.  A partial last round on a few whole warps would leave the memory
  // system idle while those finish.
  __device__ __forceinline__ int col0(int n) const {
    constexpr int nw = STRIDE / 32;
    const int rest = n % STRIDE, share = (rest + nw - 1) / nw;
    const int w = (C_ == 1 ? 0 : rank * (NT_ / 32)) + (t >> 5), l = t & 31;
    if (rest == 0) return colf();
    const int r = w * share + l;
    return l < share && r < rest ? n - rest + r : n;  // n: none in this round
  }
  __device__ __forceinline__ int colf() const { return C_ == 1 ? t : rank * NT_ + t; }
  // column of round c > 0; with ANY, n past the codeword's rounds (otherwise the
  // first round's columns would be taken a second time)
  __device__ __forceinline__ int col(int n, int c) const {
    if (ANY_ && c >= LDPCA_COLS(n, STRIDE)) return n;
    return c == 0 ? col0(n) : colf() + (c - (n % STRIDE != 0)) * STRIDE;
  }
  // barrier over the block's part
  __device__ __forceinline__ void sync() const {
    if constexpr (BLOCK)
      __syncthreads();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(NT_) : "memory");
  }
  // barrier over everything that decodes the codeword
  __device__ __forceinline__ void sync_all() const {
    if constexpr (C_ > 1)
      ld_cluster_sync();
    else
      sync();
  }
  // the value v of the leading thread (t = 0 of rank 0) in every thread,
  // through the word *w of each block; ends in no barrier, so a word is reused
  // only after a later one
  __device__ __forceinline__ int bcast(int v, int *w) const {
    if (t == 0 && rank == 0) {
      if constexpr (C_ > 1) {
#pragma unroll
        for (int b = 0; b < C_; b++) ld_st_cluster(ld_mapa((uint32_t)__cvta_generic_to_shared(w), b), (uint32_t)v);
      } else {
        *w = v;
      }
    }
    sync_all();
    return *(volatile int *)w;
  }
  // sync_all that also returns whether any thread passed p != 0; `ph`
  // alternates between calls
  __device__ __forceinline__ int sync_or(int p, LdCtl *ctl, int ph) const {
    if constexpr (C_ > 1) {
      if (__any_sync(0xffffffffu, p) && (t & 31) < C_)
        ld_st_cluster(ld_mapa((uint32_t)__cvta_generic_to_shared(&ctl->any[ph]), (uint32_t)(t & 31)), 1u);
      ld_cluster_sync();
      return (int)*(volatile uint32_t *)&ctl->any[ph];
    } else if constexpr (BLOCK) {
      return __syncthreads_or(p);
    } else {
      int r;
      asm volatile(
          "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.or.pred q, %2, %3, q;\n\tselp.s32 %0, 1, 0, q;\n\t}"
          : "=r"(r)
          : "r"(p), "r"(bar), "n"(NT_)
          : "memory");
      return r;
    }
  }
};

struct LdSmem {
  float *msg, *rowt;
  uint4 *hdr;
  uint8_t *dec, *accs;
};

__device__ __forceinline__ LdSmem ld_carve(uint8_t *base, const LadderDev &L) {
  LdSmem S;
  S.msg = reinterpret_cast<float *>(base);
  S.hdr = reinterpret_cast<uint4 *>(S.msg + L.pos_max);  // pos_max is a multiple of 4
  S.rowt = reinterpret_cast<float *>(S.hdr + L.groups);
  S.accs = reinterpret_cast<uint8_t *>(S.rowt + 32 * L.groups);  // the codeword's packed accumulated syndrome
  S.dec = reinterpret_cast<uint8_t *>(S.rowt);       // decoded bits, once BP is over
  return S;
}

// the codeword's packed accumulated syndrome (n/8 bytes, MSB first) into
// shared memory, one coalesced byte per thread, for every ladder code it tries;
// the caller synchronises before use
template <class G>
__device__ __forceinline__ void ld_stage_acc(const G &g, const uint8_t *packed, int n, uint8_t *accs) {
  constexpr int NT = G::NT;
  for (int k = g.t; k < n / 8; k += NT) accs[k] = __ldg(packed + k);
}

// fused bitplane insertion (putBitplaneToCoeff, bitplane.cpp:4-22)
template <class G>
__device__ __forceinline__ void ld_put_bitplane(const G &g, const LdpcaJob &J, const uint8_t *dec, int n) {
  constexpr int NT = G::NT;
  const int b4w = J.w >> 2, b8w = J.w >> 3;
  const int row = J.index_in_blk >> 2, col = J.index_in_blk & 3;
  for (int k = g.t; k < n; k += NT) {
    const int i = k / b4w, j = k - i * b4w;
    if (J.mode[(i >> 1) * b8w + (j >> 1)] == DVC_WZ_B) {
      int *p = J.recons_trans + ((i << 2) + row) * J.w + (j << 2) + col;
      *p = (*p << 1) + (int)dec[k];
    }
  }
}

// decoded = inv(H) * syndrome of the full-rate code (LdpcaDecoder.cpp:695-716);
// syndrome words are built in `sw` (n/32 words of shared memory).  A warp
// takes a row of the inverse at a time, its lanes consecutive words, so the
// reads (5 MB at CIF) are coalesced.
template <class G>
__device__ __forceinline__ void ld_invh_decode(const G &g, const LadderDev &L, const uint8_t *synd, uint8_t *dec,
                               uint32_t *sw) {
  constexpr int NT = G::NT;
  const int n = L.n, nw = L.invh_words, lane = g.t & 31, warp = g.t >> 5;
  for (int base = warp * 32; base < n; base += NT) {
    const int k = base + lane;
    const uint32_t b = __ballot_sync(0xffffffffu, k < n && (synd[k] & 1));
    if (lane == 0) sw[base >> 5] = b;
  }
  g.sync();
  for (int j = warp; j < n; j += NT / 32) {
    const uint32_t *row = L.invh + (size_t)j * nw;
    uint32_t x = 0;
    for (int w = lane; w < nw; w += 32) x ^= __ldg(row + w) & sw[w];
    const uint32_t odd = __ballot_sync(0xffffffffu, __popc(x) & 1);
    if (lane == 0) dec[j] = (uint8_t)(__popc(odd) & 1);
  }
  g.sync();
}

// one bit of the packed accumulated-syndrome bytes (MSB first, ByteToBit),
// from shared or global memory
__device__ __forceinline__ uint8_t ld_acc_bit(const uint8_t *packed, int i) {
  return (uint8_t)((packed[i >> 3] >> (7 - (i & 7))) & 1);
}

// bit r of the syndrome of ladder code `code` (LdpcaDecoder.cpp:684-693):
// accumulated bit idx[r % nb] + (r / nb) * period xor the same of r - 1
__device__ __forceinline__ uint32_t ld_synd_bit(const LadderDev &L, const int *idx, int nb, const uint8_t *packed,
                                                int r) {
  const int P = L.period, q = r / nb, i = r - q * nb;
  uint32_t s = ld_acc_bit(packed, __ldg(idx + i) + q * P);
  if (r > 0) s ^= ld_acc_bit(packed, i > 0 ? __ldg(idx + i - 1) + q * P : __ldg(idx + nb - 1) + (q - 1) * P);
  return s;
}

// the whole syndrome of a code in row order, one byte per row.  Thread t takes
// rows t, t + NT, ...; the quotient and remainder of a row by nb advance by
// those of NT, with no division per bit.
template <class G>
__device__ __forceinline__ void ld_build_syndrome(const G &g, const LadderDev &L, int code,
                                                  const uint8_t *packed, uint8_t *synd) {
  constexpr int NT = G::NT;
  const int m = L.synd_len[code], nb = L.bpp[code], P = L.period;
  const int *idx = L.idx + (size_t)code * P;
  const int dq = NT / nb, dr = NT - dq * nb;
  int q = g.t / nb, r = g.t - q * nb;
  for (int k = g.t; k < m; k += NT) {
    uint8_t s = ld_acc_bit(packed, __ldg(idx + r) + q * P);
    if (k > 0) s ^= ld_acc_bit(packed, r > 0 ? __ldg(idx + r - 1) + q * P : __ldg(idx + nb - 1) + (q - 1) * P);
    synd[k] = s;
    r += dr;
    q += dq;
    if (r >= nb) {
      r -= nb;
      q++;
    }
  }
}

// the full-rate code: S.dec = inv(H) * syndrome, over the staged accumulated syndrome
template <class G>
__device__ __forceinline__ void ld_full_rate(const G &g, const LadderDev &L, const LdSmem &S) {
  uint8_t *synd = reinterpret_cast<uint8_t *>(S.msg);                          // n bytes
  uint32_t *sw = reinterpret_cast<uint32_t *>(synd + ((L.n + 15) & ~15));     // then n/32 words
  ld_build_syndrome(g, L, L.num_codes - 1, S.accs, synd);
  g.sync();
  ld_invh_decode(g, L, synd, S.dec, sw);
}

// log LR of a bit (LdpcaDecoder.cpp:665-666) and its term of the entropy bound,
// (P(-log P + log(1-P)) - log(1-P)) / LOG2 with P = LR/(1+LR) (ComputeCE)
__device__ __forceinline__ float ld_entropy_term(float lr, const XlmDev &xt, const XlSmall &xs) {
  const float pco = lr / (1.0f + lr);
  const float tmp = xl_logf(xt, xs, 1.0f - pco);
  return (pco * (-xl_logf(xt, xs, pco) + tmp) - tmp) / LDPCA_LOG2;
}

// log LR of the group's columns into registers and,
// when wanted, the entropy terms into `terms` (n floats of shared memory, in a
// cluster those of its first block, whose every block has started) and the sum
// of the thread's own added to *part.  llr_in and term_in: both, when they are
// at hand.
template <class G, int MAXC>
__device__ __forceinline__ void ld_llr(const G &g, int n, const float *lr, const XlmDev &xt,
                                       const XlSmall &xs, float (&llr)[MAXC], float *terms, float *llr_out,
                                       const float *llr_in = nullptr, const float *term_in = nullptr,
                                       float *part = nullptr) {
#pragma unroll
  for (int c = 0; c < MAXC; c++) {
    const int k = g.col(n, c);
    llr[c] = 0.0f;
    if (k < n) {
      if (terms) {
        const float term = term_in ? __ldg(term_in + k) : ld_entropy_term(lr[k], xt, xs);
        if (part) *part += term;
        if constexpr (G::C > 1)
          ld_st_cluster(ld_mapa((uint32_t)__cvta_generic_to_shared(terms + k), 0), __float_as_uint(term));
        else
          terms[k] = term;
      }
      llr[c] = llr_in ? __ldg(llr_in + k) : xl_logf(xt, xs, lr[k]);
      if (llr_out) llr_out[k] = llr[c];
    }
  }
}

// the conditional-entropy bound: a sequential float sum of the terms in block
// order, divided by n (one thread; the caller synchronises before and after)
__device__ __forceinline__ float ld_entropy_sum(const float *terms, int n) {
  float h = 0.0f;
  int k = 0;
  for (; k + 8 <= n; k += 8) {
    const float v0 = terms[k], v1 = terms[k + 1], v2 = terms[k + 2], v3 = terms[k + 3];
    const float v4 = terms[k + 4], v5 = terms[k + 5], v6 = terms[k + 6], v7 = terms[k + 7];
    h += v0;
    h += v1;
    h += v2;
    h += v3;
    h += v4;
    h += v5;
    h += v6;
    h += v7;
  }
  for (; k < n; k++) h += terms[k];
  return h / (float)n;
}

// first ladder code whose rate reaches the bound (LdpcaDecoder.cpp:657-659)
__device__ __forceinline__ int ld_start_code(const LadderDev &L, float h) {
  int start = 0;
  while (start < L.num_codes - 1 && L.code_rate[start] < h) start++;
  return start;
}

// The start code from a parallel sum of the entropy terms: `part` is the sum of
// the thread's own terms.  The bound itself is a chain of n dependent float
// additions (25 K cycles at CIF, as long as a BP iteration of a lone block and
// several of a cluster's), but all a ladder needs from it is the start code.
// Adding n non-negative terms one by one in float stays within n * 2^-24 of
// their sum, so when both ends of that range (doubled for the errors of the
// parallel sum and the division) select one code, it is the code.  Returns -1
// when they do not, or when a term is not a number; every thread gets the result.
template <class G>
__device__ __forceinline__ int ld_start_near(const G &g, const LadderDev &L, float part, uint32_t *s_red, LdCtl *ctl) {
  constexpr int NW = G::NT / 32;
  const int lane = g.t & 31, warp = g.t >> 5;
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) s_red[warp] = __float_as_uint(part);
  g.sync();
  if (g.t == 0) {
    float x = 0.0f;
    for (int w = 0; w < NW; w++) x += __uint_as_float(s_red[w]);
    if constexpr (G::C > 1) {
      for (int b = 0; b < G::C; b++)
        ld_st_cluster(ld_mapa((uint32_t)__cvta_generic_to_shared(&ctl->crc[g.rank]), b), __float_as_uint(x));
    } else {
      ctl->crc[0] = __float_as_uint(x);
    }
  }
  g.sync_all();
  float h = 0.0f;
#pragma unroll
  for (int b = 0; b < G::C; b++) h += __uint_as_float(*(volatile uint32_t *)&ctl->crc[b]);
  h /= (float)L.n;
  const float err = h * ((float)L.n * 0x1p-23f);
  if (!(h >= 0.0f) || h > 1e30f) return -1;
  const int lo = ld_start_code(L, h - err), hi = ld_start_code(L, h + err);
  return lo == hi ? lo : -1;
}

// One ladder code below full rate: its syndrome (from the accumulated syndrome
// staged in S.accs by ld_stage_acc), sum-product BP until every
// parity check holds (success) or max_iter iterations ran or, when `bestp` is
// given, a lower code of the same codeword has succeeded (*bestp < code), then
// the CRC-8 of the hard decision (LdpcaDecoder.cpp:684-693, 718-758).
// Returns 1 when the code decodes with a matching CRC; `dm` then holds the
// decoded bits of the thread's columns (bit c: round c), and
// S.dec all of them (not in a cluster).  `iters` receives the BP iterations
// run.  s_ured holds NT/32 words of shared memory.
template <class G, int MAXC>
__device__ __forceinline__ int ld_try_code(const G &g, const LadderDev &L, int code, const float (&llr)[MAXC],
                           int crc, const XlmDev &xt, const uint4 *pdesc, int max_iter,
                           const volatile int *bestp, const LdSmem &S, uint32_t *s_ured, LdCtl *ctl, int &iters,
                           uint32_t &dm) {
  constexpr int NT = G::NT, C = G::C, NW = NT / 32;
  // a cluster keeps its columns' magnitudes in registers (they are stored in
  // other blocks); alone they are read back from shared memory
  constexpr bool KEEP = C > 1;
  const int n = L.n, t = g.t, lane = t & 31, warp = t >> 5;
  const int rank = C > 1 ? g.rank : 0;
  const bool lead = t == 0 && rank == 0;
  float *msg = S.msg, *rowt = S.rowt;
  const uint2 *__restrict__ grp = L.grp + (size_t)code * L.groups;
  const int ng = __ldg(L.ng + code);
  const uint32_t *__restrict__ edge = L.edge + (size_t)code * 3 * n;
  const uint32_t msg_a = (uint32_t)__cvta_generic_to_shared(msg);
  const uint32_t hdr_a = (uint32_t)__cvta_generic_to_shared(S.hdr);
  const uint32_t rowt_a = (uint32_t)__cvta_generic_to_shared(rowt);
  // an edge word: position in the low half, row slot in the high half; the
  // row's group (slot / 32) belongs to block group % C
  auto put = [&](uint32_t ed, uint32_t bits) {
    if constexpr (C > 1)
      ld_st_cluster(ld_mapa(msg_a + 4 * (ed & 0xffffu), (ed >> 21) & (C - 1)), bits);
    else
      msg[ed & 0xffffu] = __uint_as_float(bits);
  };
  auto flip = [&](uint32_t ed) {
    const uint32_t bit = 1u << ((ed >> 16) & 31u);
    if constexpr (C > 1)
      ld_xor_cluster(ld_mapa(hdr_a + 16 * (ed >> 21) + 8, (ed >> 21) & (C - 1)), bit);
    else
      atomicXor(&S.hdr[ed >> 21].z, bit);
  };
  // padding positions add +0 to their row's sum, which leaves it unchanged
  for (int p = t; p < L.pos_max / 4; p += NT) reinterpret_cast<float4 *>(msg)[p] = make_float4(0.f, 0.f, 0.f, 0.f);
  {
    const uint16_t *srow = L.slot_row + (size_t)code * 32 * L.groups;
    const int nb = L.bpp[code];
    const int *idx = L.idx + (size_t)code * L.period;
    for (int gr = rank + C * warp; gr < ng; gr += C * NW) {
      const uint2 place = __ldg(grp + gr);
      const uint32_t b = __ballot_sync(
          0xffffffffu, lane < (int)place.y && ld_synd_bit(L, idx, nb, S.accs, __ldg(srow + 32 * gr + lane)));
      if (lane == 0) S.hdr[gr] = make_uint4(place.x, b, b, place.y);
    }
  }
  if (t == 0) {
    ctl->any[0] = ctl->any[1] = 0;
    ctl->stop = 0;
  }
  uint32_t mg[KEEP ? MAXC : 1][3];
  g.sync_all();
  // first magnitudes: phi(|LLR|) on the three edges of each column
#pragma unroll(KEEP ? MAXC : 2)
  for (int c = 0; c < MAXC; c++) {
    const int k = g.col(n, c);
    if (k < n) {
      const float l = llr[c];
      const uint32_t bits = (__float_as_uint(xl_phi(xt, pdesc, (fabsf(l) + 1e-9f) / 2.0f)) & 0x7fffffffu) |
                            (__float_as_uint(l) & 0x80000000u);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        put(__ldg(edge + i * n + k), bits);
        if constexpr (KEEP) mg[c][i] = bits;
      }
    }
  }
  // the edge words and the LLR of the next column are read one round ahead
  // (round 0's during the row pass)
  uint32_t nx[3];
  float nl = llr[0];
  const int kfirst = g.col0(n);
#pragma unroll
  for (int i = 0; i < 3; i++) nx[i] = ld_edge(edge + i * n + min(kfirst, n - 1));
  dm = 0;
  int best = bestp && lead ? *bestp : LDPCA_NONE;
  g.sync_all();
  bool converged = false;
  int it = 0;
  for (;;) {
    // rows: lane l of a warp sums the row in slot 32 g + l of its groups.  The
    // loads of four edges are issued before their adds, which stay in edge
    // order; with groups of 3 to 7 edges at the higher codes the pass is bound
    // by its instructions, so full groups take constant strides
    int wrong = 0;
    for (int gr = rank + C * warp; gr < ng; gr += C * NW) {
      const uint4 hd = S.hdr[gr];
      const float *p = msg + (hd.x & 0xffffu) + lane;
      const int deg = (int)(hd.x >> 16);
      float s = 0.0f;
      uint32_t x = (hd.y >> lane) << 31;  // xor of the signs and the syndrome bit, in the top bit
      auto add = [&](float v) {
        s += fabsf(v);
        x ^= __float_as_uint(v);
      };
      auto row = [&](int width) {
        int left = deg;
        for (; left >= 4; left -= 4, p += 4 * width) {
          const float v0 = p[0], v1 = p[width], v2 = p[2 * width], v3 = p[3 * width];
          add(v0);
          add(v1);
          add(v2);
          add(v3);
        }
        if (left >= 2) {
          const float v0 = p[0], v1 = p[width];
          add(v0);
          add(v1);
          p += 2 * width;
        }
        if (left & 1) add(p[0]);
      };
      const int width = (int)hd.w;
      if (width == 32)
        row(32);
      else if (lane < width)
        row(width);
      const uint32_t r = __float_as_uint(s) | (x & 0x80000000u);
      if (lane < width) {
        if constexpr (C > 1) {
#pragma unroll
          for (int b = 0; b < C; b++) ld_st_cluster(ld_mapa(rowt_a + 4 * (32 * gr + lane), b), r);
        } else {
          rowt[32 * gr + lane] = __uint_as_float(r);
        }
      }
      wrong |= (int)(hd.z != 0);
    }
    if (lead && best < code) {
      if constexpr (C > 1) {
#pragma unroll
        for (int b = 0; b < C; b++) ld_st_cluster(ld_mapa((uint32_t)__cvta_generic_to_shared(&ctl->stop), b), 1u);
      } else {
        ctl->stop = 1;
      }
    }
    const int any_wrong = g.sync_or(wrong, ctl, it & 1);
    if (it > 0 && !any_wrong) {
      converged = true;
      break;
    }
    // abandon a code above a known success
    if (it == max_iter || *(volatile uint32_t *)&ctl->stop) break;
    if (C > 1 && t == 0) ctl->any[(it & 1) ^ 1] = 0;  // last read before the previous edge pass
    it++;
    if (bestp && lead) best = *bestp;  // arrives during the edge pass, used after it
    // edges, column by column (a rolled loop: seven copies of it would not
    // stay in the instruction cache)
    int k = kfirst;
#pragma unroll(KEEP ? MAXC : 1)
    for (int c = 0; c < MAXC; c++) {
      const int kn = c + 1 < MAXC ? g.col(n, c + 1) : kfirst;
      uint32_t ed[3], mv[3];
      const float l = nl;
#pragma unroll
      for (int i = 0; i < 3; i++) ed[i] = nx[i];
#pragma unroll
      for (int i = 0; i < 3; i++) nx[i] = ld_edge(edge + i * n + min(kn, n - 1));
      nl = llr[c + 1 < MAXC ? c + 1 : 0];
      if (k < n) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const uint32_t r = __float_as_uint(rowt[ed[i] >> 16]);
          const uint32_t a = KEEP ? mg[KEEP ? c : 0][i] : __float_as_uint(msg[ed[i] & 0xffffu]);
          // c->v: phi(row sum - own magnitude) with the product of the other signs
          const float y = (fabsf(__uint_as_float(r)) - fabsf(__uint_as_float(a)) + 1e-9f) / 2.0f;
          mv[i] = __float_as_uint(xl_phi(xt, pdesc, y)) ^ ((r ^ a) & 0x80000000u);
        }
        // total in edge order, hard decision, extrinsic messages and their
        // magnitudes for the next iteration
        float tot = l;
#pragma unroll
        for (int i = 0; i < 3; i++) tot += __uint_as_float(mv[i]);
        if ((__float_as_uint(tot) >> 31) != ((dm >> c) & 1u)) {
          dm ^= 1u << c;
#pragma unroll
          for (int i = 0; i < 3; i++) flip(ed[i]);
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const float v = tot - __uint_as_float(mv[i]);
          mv[i] = (__float_as_uint(xl_phi(xt, pdesc, (fabsf(v) + 1e-9f) / 2.0f)) & 0x7fffffffu) |
                  (__float_as_uint(v) & 0x80000000u);
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          put(ed[i], mv[i]);
          if constexpr (KEEP) mg[c][i] = mv[i];
        }
      }
      k = kn;
    }
    g.sync_all();
  }
  iters = it;
  if (!converged) {
    g.sync_all();  // every thread has read ctl: the caller may reuse it
    return 0;
  }
  // the hard decisions into dec, and the CRC-8 of the decoded bitplane as the
  // xor of single-bit CRCs (the CRC is linear for a fixed length with zero
  // initial value and no final xor)
  uint32_t cr = 0;
  for (int c = 0; c < MAXC; c++) {
    const int k = g.col(n, c);
    if (k < n) {
      const uint32_t d = (dm >> c) & 1u;
      if constexpr (C == 1) S.dec[k] = (uint8_t)d;
      if (d) cr ^= __ldg(L.crc_tab + k);
    }
  }
  for (int o = 16; o > 0; o >>= 1) cr ^= __shfl_xor_sync(0xffffffffu, cr, o);
  if (lane == 0) s_ured[warp] = cr;
  g.sync();
  if (t == 0) {
    uint32_t x = 0;
    for (int w = 0; w < NW; w++) x ^= s_ured[w];
    if constexpr (C > 1) {
      for (int b = 0; b < C; b++) ld_st_cluster(ld_mapa((uint32_t)__cvta_generic_to_shared(&ctl->crc[rank]), b), x);
    } else {
      ctl->flag = (int)(x & 0xffu) == crc;
    }
  }
  g.sync_all();
  int ok;
  if constexpr (C > 1) {
    uint32_t x = 0;
#pragma unroll
    for (int b = 0; b < C; b++) x ^= *(volatile uint32_t *)&ctl->crc[b];
    ok = (int)(x & 0xffu) == crc;
  } else {
    ok = ctl->flag;
  }
  g.sync_all();
  return ok;
}

}  // namespace dvc
