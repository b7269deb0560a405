// Test driver: the library's host code (dispatch, buffers, streams) linked with
// a CUDA runtime that runs no kernel.  Device memory is host memory, a launch is
// checked as the runtime checks it (a function's dynamic shared memory against
// the attribute set for it) and written down, and allocations can be made to
// fail by size.  tests/test_host_routes.py builds it from the library's object
// files and reads what it prints.  The C-library table sweeps are left out (the
// kernels that read the tables do not run).
#include <cuda_runtime.h>
#include <sys/resource.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "context.h"
#include "dvc_b200.h"
#include "libm_tables.h"

namespace dvc {
Context *context_of(dvc_ctx *ctx);
}

// ------------------------------------------------------------ the runtime
namespace {
std::map<const void *, std::string> g_name;   // host stub -> kernel
std::map<const void *, size_t> g_smem;        // largest dynamic shared memory allowed
std::map<void *, size_t> g_mem;               // device allocations
size_t g_live = 0, g_fail_from = ~(size_t)0;  // bytes held; allocations of this size and more fail
int g_fail_after = 0;                         // ... but for the first few
int g_streams = 0, g_events = 0;              // alive
bool g_record = false;
cudaError_t g_last = cudaSuccess;

cudaError_t take(void **p, size_t bytes) {
  *p = nullptr;
  if ((bytes >= g_fail_from && g_fail_after-- <= 0) || bytes > ((size_t)1 << 36)) return g_last = cudaErrorMemoryAllocation;
  *p = aligned_alloc(256, (bytes + 255) & ~(size_t)255);
  memset(*p, 0, bytes);
  g_mem[*p] = bytes;
  g_live += bytes;
  return cudaSuccess;
}
cudaError_t give(void *p) {
  if (!p) return cudaSuccess;
  auto it = g_mem.find(p);
  if (it == g_mem.end()) return cudaErrorInvalidValue;
  g_live -= it->second;
  g_mem.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t launch(const void *f, dim3 grid, dim3 block, unsigned cluster, size_t smem) {
  const size_t most = g_smem.count(f) ? g_smem[f] : 48 * 1024;
  const bool bad = smem > most || grid.x % cluster != 0 || block.x > 1024;
  if (g_record)
    printf("launch %s grid %u block %u cluster %u smem %zu%s\n", g_name[f].c_str(), grid.x, block.x, cluster, smem,
           bad ? " refused" : "");
  return bad ? cudaErrorInvalidValue : cudaSuccess;
}
struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_call;
}  // namespace

extern "C" {
void **__cudaRegisterFatBinary(void *) { return (void **)&g_call; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  g_name[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  g_call = {g, b, s, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = g_call.grid;
  *b = g_call.block;
  *s = g_call.smem;
  *(cudaStream_t *)st = g_call.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t smem, cudaStream_t) {
  return launch(f, g, b, 1, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  unsigned cluster = 1;
  for (unsigned i = 0; i < c->numAttrs; i++)
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
  return launch(f, c->gridDim, c->blockDim, cluster, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > 227 * 1024) return cudaErrorInvalidValue;
    g_smem[f] = (size_t)v;
  }
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void **p, size_t n) { return (*p = calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static char room[1 << 20];
  *p = room;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t) new int(0);
  g_streams++;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  delete (int *)s;
  g_streams--;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t) new int(0);
  g_events++;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (int *)e;
  g_events--;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1 << 27;
  return cudaSuccess;
}
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) {
  *p = nullptr;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaCreateTextureObject(cudaTextureObject_t *t, const cudaResourceDesc *, const cudaTextureDesc *,
                                    const cudaResourceViewDesc *) {
  *t = 1;
  return cudaSuccess;
}
cudaError_t cudaDestroyTextureObject(cudaTextureObject_t) { return cudaSuccess; }
cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f) {
  return {x, y, z, w, f};
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "CUDA error"; }

int dvc_libm_build(const char *, int, char *, int) { return 0; }
}

int dvc_libm_load(const char *, XlmHost *out, char *, int) {
  out->log_tab.assign(4, 0);
  out->exp_tab.assign(4, 0);
  memset(&out->hdr, 0, sizeof out->hdr);
  out->hdr.log_cap = out->hdr.exp_cap = 2;
  out->hdr.tanh_y1 = 16;
  return 0;
}
void dvc_phi_build(float *, uint32_t, uint32_t, int) {}
bool dvc_phi_pack(const float *, uint32_t, uint32_t, int, PhiPacked &out, char *, int) {
  out.desc.assign(4, 0);
  out.rec.assign(4, 0);
  return true;
}

// ---------------------------------------------------------------- the modes
static dvc_ctx *context(const char *data, const char *tables) {
  dvc_ctx *c = nullptr;
  const int rc = dvc_create(data, tables, 0, &c);
  if (rc != DVC_OK) {
    printf("create %d %s\n", rc, dvc_last_error(c));
    exit(0);
  }
  return c;
}

// one dvc_ldpca_decode of `count` codewords of zeros
static int decode_zeros(dvc_ctx *c, int n, int count) {
  std::vector<float> lr((size_t)count * n, 1.0f), ent(count);
  std::vector<uint8_t> acc((size_t)count * n / 8), crc(count), dec((size_t)count * n);
  std::vector<int> res((size_t)count * 4);
  return dvc_ldpca_decode(c, n, count, lr.data(), acc.data(), crc.data(), dec.data(), res.data(), ent.data(), 50);
}

// files DATA TABLES DATA2: codewords of both lengths and a batch of them with one
// ladder file after another
static void files(char **a) {
  for (const char *data : {a[0], a[2]}) {
    dvc_ctx *c = context(data, a[1]);
    g_record = true;
    for (int n : {1584, 6336})
      for (int count : {1, 200, 600}) printf("rc %d\n", decode_zeros(c, n, count));
    g_record = false;
    dvc_destroy(c);
  }
}

// the reference-shaped call on zeros
static int decoder_zeros(dvc_ctx *c, int n) {
  std::vector<float> lr(n, 1.0f);
  std::vector<uint8_t> acc(n), dec(n);
  int rate = 0;
  return dvc_LdpcaDecoder(c, n, lr.data(), acc.data(), dec.data(), &rate, 0, 0.5f);
}

// decode DATA TABLES n count
static void decode(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  g_record = true;
  printf("rc %d\n", decode_zeros(c, atoi(a[2]), atoi(a[3])));
  g_record = false;
  dvc_destroy(c);
}

// scarce DATA TABLES n count from after: the two LDPCA calls while allocations
// of `from` bytes and more, but for the first `after`, are refused, then with memory
static void scarce(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  const int n = atoi(a[2]), count = atoi(a[3]);
  g_record = true;
  for (int turn = 0; turn < 2; turn++) {
    g_fail_from = turn == 0 ? strtoull(a[4], nullptr, 0) : ~(size_t)0;
    g_fail_after = atoi(a[5]);
    const int rc = count > 0 ? decode_zeros(c, n, count) : decoder_zeros(c, n);
    printf("rc %d last %d\n", rc, (int)cudaGetLastError());
  }
  g_record = false;
  dvc_destroy(c);
}

// huge DATA TABLES n count: a count that no device holds (the inputs are not read)
static void huge(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  const int n = atoi(a[2]), count = atoi(a[3]);
  const rlimit most = {(rlim_t)3 << 30, (rlim_t)3 << 30};
  setrlimit(RLIMIT_AS, &most);
  g_fail_from = (size_t)1 << 30;
  float lr = 1.0f;
  uint8_t acc = 0, crc = 0;
  int res[4] = {0};
  printf("rc %d\n", dvc_ldpca_decode(c, n, count, &lr, &acc, &crc, nullptr, res, nullptr, 50));
  dvc_destroy(c);
}

// a frame of zeros between two references
struct Frame {
  std::vector<uint8_t> past, future, crc, acc, recon;
  int range[16];
  dvc_wz_frame f;
  Frame(int w, int h, int q) : past(w * h), future(w * h), crc(64), acc(64 * w * h / 128), recon(w * h) {
    for (int &r : range) r = 100;
    memset(&f, 0, sizeof f);
    f.width = w;
    f.height = h;
    f.qindex = q;
    f.cur_idx = 1;
    f.future_idx = 2;
    f.past = past.data();
    f.future = future.data();
    f.crc = crc.data();
    f.acc_synd = acc.data();
    f.recon = recon.data();
    f.ac_range = range;
  }
};

// session DATA TABLES sequences levels max_batch streams: what a session of QCIF
// sequences holds, and two runs of it; a sequence is a GOP of 2^levels frames,
// whose first level is the middle frame, the next those half way to its ends
static void session(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  const int sequences = atoi(a[2]), levels = atoi(a[3]), gop = 1 << levels, count = sequences * (gop - 1);
  const int s0 = g_streams;
  std::vector<Frame> frames;
  std::vector<dvc_wz_frame> list;
  frames.reserve(count);
  for (int i = 0; i < count; i++) frames.emplace_back(176, 144, 1);
  for (int i = 0; i < count; i++) {
    const int at = i % (gop - 1) + 1, half = at & -at;  // frame `at` lies between at - half and at + half
    dvc_wz_frame f = frames[i].f;
    if (at - half > 0) f.past = frames[i - half].recon.data();
    if (at + half < gop) f.future = frames[i + half].recon.data();
    list.push_back(f);
  }
  dvc_session *s = nullptr;
  int rc = dvc_session_create(c, count, list.data(), atoi(a[4]), atoi(a[5]), &s);
  printf("rc %d\nstreams %d\n", rc, g_streams - s0);
  double ms = 0;
  for (int run = 0; run < 2; run++) printf("rc %d\n", dvc_session_run(s, 0, &ms));
  dvc_session_destroy(s);
  dvc_destroy(c);
}

// server DATA TABLES w h q range count: the bytes a server charges for requests in
// flight, and those its cohort of them holds on the device
static void server(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  const int w = atoi(a[2]), h = atoi(a[3]), q = atoi(a[4]), count = atoi(a[6]);
  dvc_server *s = nullptr;
  printf("rc %d\n", dvc_server_create(c, (size_t)64 << 30, 1, count, &s));
  const size_t before = g_live;
  long long ticket, pending, in_flight;
  size_t charged = 0;
  int done = 0;
  for (int i = 0; i < count; i++) {
    Frame f(w, h, q);
    for (int &r : f.range) r = atoi(a[5]);
    printf("rc %d\n", dvc_server_submit(s, &f.f, &ticket));
  }
  printf("rc %d\n", dvc_server_poll(s, &done));
  dvc_server_stats(s, &pending, &in_flight, &charged);
  printf("in flight %lld charged %zu held %zu\n", in_flight, charged, g_live - before);
  dvc_server_destroy(s);
  dvc_destroy(c);
}

// shapes DATA TABLES: a frame, and codewords of both lengths a block each
static void shapes(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  Frame f(176, 144, 1);
  g_record = true;
  printf("rc %d\n", dvc_decode_wz_frames(c, 1, &f.f));
  void *room = nullptr;  // no kernel reads it
  cudaMalloc(&room, 1 << 16);
  for (int n : {1584, 6336})
    printf("rc %d\n", dvc_ldpca_decode_noalloc(c, n, 1, (float *)room, (uint8_t *)room, (uint8_t *)room, nullptr,
                                               (int *)room, nullptr, 50, nullptr));
  g_record = false;
  cudaFree(room);
  dvc_destroy(c);
}

// layout DATA TABLES: the BP layout of every code of a ladder file.  Every edge has
// a position of its own inside its row's group, a row's edges follow one another
// in edge order, and its slot names the row, found here from the file's data.
static void layout(char **a) {
  dvc_ctx *c = context(a[0], a[1]);
  for (const dvc::LadderHost &L : dvc::context_of(c)->ladders_host) {
    int bad = 0, most = 0;
    for (int code = 0; code < L.num_codes; code++) {
      const int b = L.bpp[code], m = L.synd_len[code];
      std::vector<int> next(m, 0), used(L.pos_max, 0), rows(m, 0);
      int positions = 0, held = 0;
      for (int g = 0; g < L.ng[code]; g++) {
        const uint2 p = L.grp[(size_t)code * L.groups + g];
        bad += p.y < 1 || p.y > 32;
        for (uint32_t l = 0; l < p.y; l++) rows[L.slot_row[((size_t)code * L.groups + g) * 32 + l]]++;
        positions += (int)((p.x >> 16) * p.y);
        held += (int)p.y;
      }
      for (int r = 0; r < m; r++) bad += rows[r] != 1;
      bad += held != m || positions > L.pos_max;
      most = std::max(most, positions);
      for (int k = 0; k < L.n; k++)
        for (int i = 0; i < 3; i++) {
          int r = 0;  // the first kept position at or after the edge's full-rate row
          const int at = L.ir_full[3 * k + i], q = at / L.period;
          while (r < b && L.idx[(size_t)code * L.period + r] < at - q * L.period) r++;
          r += q * b;
          const uint32_t e = L.edge[((size_t)code * 3 + i) * L.n + k], p = e & 0xffffu, s = e >> 16;
          if ((int)(s >> 5) >= L.ng[code] || (int)p >= L.pos_max) {
            bad++;
            continue;
          }
          const uint2 G = L.grp[(size_t)code * L.groups + (s >> 5)];
          bad += (s & 31) >= G.y || L.slot_row[(size_t)code * L.groups * 32 + s] != r;
          const int nth = next[r]++;
          bad += p != (G.x & 0xffffu) + (uint32_t)nth * G.y + (s & 31) || nth >= (int)(G.x >> 16) || used[p]++;
        }
    }
    printf("length %d codes %d positions %d groups %d bad %d\n", L.n, L.num_codes, most, L.groups, bad);
  }
  dvc_destroy(c);
}

int main(int argc, char **argv) {
  const std::string mode = argc > 1 ? argv[1] : "";
  if (mode == "files" && argc == 5) files(argv + 2);
  else if (mode == "decode" && argc == 6) decode(argv + 2);
  else if (mode == "scarce" && argc == 8) scarce(argv + 2);
  else if (mode == "huge" && argc == 6) huge(argv + 2);
  else if (mode == "session" && argc == 8) session(argv + 2);
  else if (mode == "server" && argc == 9) server(argv + 2);
  else if (mode == "shapes" && argc == 4) shapes(argv + 2);
  else if (mode == "layout" && argc == 4) layout(argv + 2);
  else return 2;
  printf("left bytes %zu streams %d events %d\n", g_live, g_streams, g_events);
  return 0;
}
