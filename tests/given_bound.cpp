// Test driver: the block-per-ladder form of the LDPCA kernel with the bound given,
// which the entry points reach only for calls that cannot use speculative slots.
//   given_bound DATA TABLES n count lr.f32 acc.u8 crc.u8
// decodes the codewords with dvc_ldpca_decode, then with launch_ldpca and the
// bounds that call reported, and compares everything.  Exit status 0: equal.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "context.h"
#include "dvc_b200.h"
#include "kernels.h"

namespace dvc {
Context *context_of(dvc_ctx *ctx);
}

template <class T>
static std::vector<T> file(const char *path, size_t n) {
  std::vector<T> v(n);
  FILE *f = fopen(path, "rb");
  if (!f || fread(v.data(), sizeof(T), n, f) != n) exit(3);
  fclose(f);
  return v;
}

template <class T>
static T *dev(const T *h, size_t n) {
  T *p = nullptr;
  if (cudaMalloc((void **)&p, n * sizeof(T)) != cudaSuccess) exit(4);
  if (h ? cudaMemcpy(p, h, n * sizeof(T), cudaMemcpyHostToDevice) : cudaMemset(p, 0xEE, n * sizeof(T))) exit(4);
  return p;
}

int main(int argc, char **argv) {
  if (argc != 8) return 2;
  const int n = atoi(argv[3]), count = atoi(argv[4]);
  const size_t nb = n / 8;
  const auto lr = file<float>(argv[5], (size_t)count * n);
  const auto acc = file<uint8_t>(argv[6], count * nb), crc = file<uint8_t>(argv[7], count);
  dvc_ctx *ctx = nullptr;
  if (dvc_create(argv[1], argv[2], 0, &ctx) != DVC_OK) return 5;
  std::vector<uint8_t> dec((size_t)count * n), dec2(dec.size());
  std::vector<int> res((size_t)count * 4), res2(res.size());
  std::vector<float> ent(count), ent2(count);
  if (dvc_ldpca_decode(ctx, n, count, lr.data(), acc.data(), crc.data(), dec.data(), res.data(), ent.data(), 50)) return 6;
  dvc::Context &c = *dvc::context_of(ctx);
  float *d_lr = dev(lr.data(), lr.size()), *d_ent = dev<float>(nullptr, count);
  uint8_t *d_acc = dev(acc.data(), acc.size()), *d_dec = dev<uint8_t>(nullptr, dec.size());
  int *d_res = dev<int>(nullptr, res.size());
  std::vector<dvc::LdpcaJob> jobs(count);
  for (int i = 0; i < count; i++) {
    dvc::LdpcaJob &j = jobs[i];
    memset(&j, 0, sizeof j);
    j.active = 1;
    j.lr = d_lr + (size_t)i * n;
    j.acc = d_acc + i * nb;
    j.crc = crc[i];
    j.decoded = d_dec + (size_t)i * n;
    j.result = d_res + 4 * i;
    j.entropy = d_ent + i;
    j.use_given_entropy = 1;
    j.given_entropy = ent[i];
  }
  dvc::LdpcaJob *d_jobs = dev(jobs.data(), jobs.size());
  int bad = 0;
  for (int turn = 0; turn < 3; turn++) {
    if (dvc::launch_ldpca(*c.ladder(n), d_jobs, count, c.xlm, 50, c.stream) != cudaSuccess) return 7;
    if (cudaStreamSynchronize(c.stream) != cudaSuccess) return 8;
    if (cudaMemcpy(dec2.data(), d_dec, dec2.size(), cudaMemcpyDeviceToHost) ||
        cudaMemcpy(res2.data(), d_res, res2.size() * 4, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(ent2.data(), d_ent, count * 4, cudaMemcpyDeviceToHost))
      return 8;
    bad |= (dec != dec2) | (res != res2) << 1 | (memcmp(ent.data(), ent2.data(), count * 4) != 0) << 2;
  }
  dvc_destroy(ctx);
  printf("bits %s, results %s, bounds %s\n", bad & 1 ? "differ" : "equal", bad & 2 ? "differ" : "equal",
         bad & 4 ? "differ" : "equal");
  return bad ? 1 : 0;
}
