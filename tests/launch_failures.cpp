// Launches of the training entry points that fail, without a GPU: this program brings its own CUDA runtime
// calls, which count and, at a chosen place, answer with an error that cudaGetLastError returns once.  Every
// such error has to come back from the entry point.  Prints one line per error that did not.
// Argument: which case.  One process per case, because kernels are opted in once per process and device.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "bnb_trunk.h"

namespace {
int device = 0, last = 0, launches = 0, fail_launch = -1, opt_ins = 0, fail_opt_in = -1, copies = 0, fail_copy = -1;
bool failed = false;
int answer(int& count, int fail) {
  if (count++ != fail) return 0;
  failed = true;
  last = 719;
  return last;
}
void begin(int launch, int opt_in, int copy) {
  last = launches = opt_ins = copies = 0;
  failed = false;
  fail_launch = launch; fail_opt_in = opt_in; fail_copy = copy;
  device = (device + 1) % 64;   // a new device for the first 63 calls of the process
}
}  // namespace

extern "C" {
unsigned __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
int cudaLaunchKernel() { return answer(launches, fail_launch); }
int cudaLaunchKernelExC() { return answer(launches, fail_launch); }
int cudaFuncSetAttribute() { return answer(opt_ins, fail_opt_in); }
int cudaMemsetAsync() { return answer(copies, fail_copy); }
int cudaMemcpyAsync() { return answer(copies, fail_copy); }
int cudaGetLastError() { const int e = last; last = 0; return e; }
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int* v) { *v = 148; return 0; }
int cudaHostAlloc(void** p, size_t n) { *p = std::calloc(1, n); return 0; }
int cudaStreamIsCapturing(void*, int* c) { *c = 0; return 0; }
}

namespace {

struct Case { const char* name; int d_model, ships, fields, bullets, precision, blocks; };

// Never read on the host: an address of the right alignment, and space behind it as far as the calls are told.
float* nowhere() {
  static uintptr_t at = 1u << 20;
  return reinterpret_cast<float*>(at += 1u << 20);
}
constexpr size_t plenty = size_t(1) << 40;

int swallowed = 0;
template <class F>
void check(const Case& c, const char* what, F call) {
  begin(-1, -1, -1);
  if (const int st = call()) { std::printf("%s %s: status %d without a failure\n", c.name, what, st); ++swallowed; return; }
  const int n[3] = {launches, opt_ins, copies};
  begin(-1, -1, -1);
  (void)call();
  if (opt_ins != n[1]) { std::printf("%s %s: %d opt-ins on the first device, %d on the second\n", c.name, what, n[1], opt_ins); ++swallowed; }
  if (n[0] == 0 && n[2] == 0) { std::printf("%s %s: nothing was launched\n", c.name, what); ++swallowed; }
  const char* kind[3] = {"launch", "opt-in", "copy"};
  for (int k : {1, 0, 2})   // opt-ins first: their devices have to be new
    for (int i = 0; i < n[k]; ++i) {
      begin(k == 0 ? i : -1, k == 1 ? i : -1, k == 2 ? i : -1);
      const int st = call();
      if (!failed) continue;   // an opt-in that is made once
      if (st != BNB_ERR_LAUNCH) { std::printf("%s %s: failed %s %d of %d is not reported\n", c.name, what, kind[k], i, n[k]); ++swallowed; }
      if (last) { std::printf("%s %s: failed %s %d leaves its error to the next call\n", c.name, what, kind[k], i); ++swallowed; }
    }
}

void run(const Case& c, int stage) {
  const int T = 3, B = 5, tokens = c.ships + c.fields, per_block = 2;
  BnbBatch b{};
  b.n_envs = B;
  b.tokens_per_env = b.max_tokens_per_env = tokens;
  b.ships_per_env = c.ships;
  b.total_tokens = B * tokens;
  b.total_ships = B * c.ships;
  std::vector<BnbSpatialWeights> sw((size_t)c.blocks * per_block);
  std::vector<BnbTemporalWeights> tw((size_t)c.blocks);
  std::vector<BnbSpatialGrads> sg(sw.size());
  std::vector<BnbTemporalGrads> tg(tw.size());
  auto fill = [](auto& s, size_t n) {   // rows of float*
    float** f = reinterpret_cast<float**>(&s);
    for (size_t i = 0; i < n; ++i) f[i] = nowhere();
  };
  for (size_t i = 0; i < sw.size(); ++i) {
    const size_t n = c.bullets && i % per_block == 0 ? 9 : 7;
    fill(sw[i], n);
    fill(sg[i], n);
  }
  for (size_t i = 0; i < tw.size(); ++i) {
    fill(tw[i], c.fields ? 16 : 15);
    fill(tg[i], c.fields ? 16 : 15);
  }
  BnbBullets bul{};
  bul.tokens = nowhere();
  bul.active = reinterpret_cast<const uint8_t*>(nowhere());
  bul.per_env = c.bullets;
  const BnbBullets* bp = c.bullets ? &bul : nullptr;
  float *x = nowhere(), *y = nowhere(), *hin = nowhere(), *hout = nowhere(), *dy = nowhere(), *dx = nowhere(), *dh = nowhere(), *db = nowhere();
  const uint8_t *alive = reinterpret_cast<const uint8_t*>(nowhere()), *done = reinterpret_cast<const uint8_t*>(nowhere());
  void *kept = nowhere(), *scratch = nowhere();
  if (stage == 0)
    check(c, "forward", [&] {
      return bnb_trunk_sequence_fwd_train(sw.data(), tw.data(), c.blocks, per_block, 1, c.d_model, 4, x, alive, bp, y, hin, hout, done, &b, T,
                                          c.precision, kept, plenty, scratch, plenty, nullptr);
    });
  void* k = stage == 1 ? kept : nullptr;
  if (stage > 0)
    check(c, k ? "backward" : "backward that recomputes", [&] {
      return bnb_trunk_sequence_bwd(sw.data(), tw.data(), sg.data(), tg.data(), c.blocks, per_block, 1, c.d_model, 4, x, alive, bp, hin, done,
                                    &b, T, c.precision, dy, hout, dx, dh, c.bullets ? db : nullptr, k, k ? plenty : 0, scratch, plenty, nullptr);
    });
}

}  // namespace

int main(int argc, char** argv) {
  const Case cases[] = {{"bf16 ships", 128, 8, 0, 0, BNB_BF16, 2},      {"bf16 fields bullets", 128, 8, 4, 80, BNB_BF16, 2},
                        {"bf16 fleet", 128, 40, 3, 50, BNB_BF16, 1},    {"bf16 narrow", 64, 8, 2, 5, BNB_BF16, 1},
                        {"float32 bullets", 128, 8, 4, 12, BNB_FP32, 1}, {"no sublayers", 128, 8, 0, 0, BNB_FP32, 0}};
  const int which = argc > 1 ? std::atoi(argv[1]) : -1;
  if (which < 0 || which >= 18) return 2;
  run(cases[which / 3], which % 3);
  return swallowed != 0;
}
