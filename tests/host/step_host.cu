// The host side of stepping (fsl_group.cu) against a CUDA runtime that does
// nothing but count (counting_cudart.cpp), so that refused calls can be made
// on the CPU; the launchers of the kernels are defined here.
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "../../fluam_b200/csrc/fsl_group.cu"

extern cudaError_t g_last;  // the runtime's last error (counting_cudart.cpp)
extern int g_launched;      // graphs launched
extern char *g_pin, *g_pin_dev;  // the one page-locked range
extern size_t g_pin_bytes;
static int g_refuse = 0;    // the next launches of the noise that are refused

#define CHECK(c)                                                 \
  do {                                                           \
    if (!(c)) {                                                  \
      std::printf("line %d: %s\n", __LINE__, #c);                \
      return 1;                                                  \
    }                                                            \
  } while (0)

namespace fsl {
struct FftPlan {};
FftPlan* fft_plan_create(const Params&) { return new FftPlan(); }
void fft_plan_destroy(FftPlan* f) { delete f; }
void fft_autotune(FftPlan*, const Batch&, cudaStream_t) {}
void fft_tuning(const FftPlan*, FftTuning& t) { t = FftTuning{}; }
const GPlan* fft_general(const FftPlan*) { return nullptr; }
bool solve_clears_field(const Batch&, const FftPlan*) { return true; }
bool tile_eligible(const Params&) { return false; }
void tile_init() {}
bool block_lists(const Batch&) { return false; }
bool block_lists_eligible(const Batch&) { return false; }
int block_lists_env() { return -1; }
void lists_autotune(const Batch&, cudaStream_t, float*) {}
void launch_noise(const Batch&, cudaStream_t, int, int) {
  if (g_refuse > 0) {
    --g_refuse;
    g_last = cudaErrorInvalidConfiguration;
  }
}
cudaError_t launch_pair_lists(const Batch&, int, cudaStream_t) { return cudaSuccess; }
void launch_cells(const Batch&, int, cudaStream_t, bool) {}
void launch_forces(const Batch&, int, cudaStream_t, bool) {}
void launch_spread(const Batch&, int, int, cudaStream_t, bool, bool) {}
void launch_spread_w(const Batch&, int, int, double, cudaStream_t) {}
void launch_solve(const Batch&, FftPlan*, int, double, int, cudaStream_t, Prof*, cudaEvent_t) {}
void launch_interp_update(const Batch&, int, cudaStream_t, bool) {}
void launch_observe(const Batch&, cudaStream_t) {}
void launch_step_counter(const Batch&, cudaStream_t) {}
void launch_field_clear(const Batch&, cudaStream_t) {}
void launch_moved_check(const Rep&, cudaStream_t) {}
void launch_reset_lists(const Rep&, cudaStream_t) {}
void launch_io_in(const Rep&, const double*, cudaStream_t) {}
void launch_io_out(const Rep&, double*, cudaStream_t) {}
void launch_inc_w(const Batch&, int, cudaStream_t) {}
int launch_g_forward(const Batch&, const GPlan*, int, cudaStream_t) { return 0; }
int launch_g_inverse(const Batch&, const GPlan*, int, int, double, cudaStream_t) { return 0; }
void launch_g_z(const Batch&, const GPlan*, int, cudaStream_t) {}
void launch_q2_field(const Batch&, cudaStream_t, Prof*) {}
void launch_q2_forces(const Batch&, cudaStream_t) {}
void launch_q2_solve(const Batch&, const GPlan*, cudaStream_t, Prof*) {}
int launch_q2_update(const Batch&, int, cudaStream_t) { return 0; }
}  // namespace fsl

using namespace fsl;

// A class of one instance with n particles in a box of m cells a side.
struct One {
  Params P;
  Slot slot;
  Group g;
  int make(int m, int n) {
    fsl_config c{};
    c.mx = c.my = c.mz = m;
    c.lx = c.ly = c.lz = m;
    c.shearviscosity = 1;
    c.dt = 0.01;
    c.kernel = 3;
    std::vector<double> q(3 * (size_t)n, 0.25);
    if (make_params(c, n, P) || group_init(g, P) || slot_alloc(slot, P, n, nullptr) || slot_reset(slot, P, q.data(), c, nullptr)) return 1;
    g.slots.push_back(&slot);
    return 0;
  }
  ~One() {
    group_destroy(g);
    slot_free(slot);
  }
};

// A launch refused while a step is captured: an error and no graph, and the
// step again once launches are accepted.
static int refused(bool each) {
  One a, b;
  CHECK(a.make(8, 3) == 0 && b.make(10, 4) == 0);
  Exec e;
  CHECK(exec_init(e, 0) == 0);
  auto step = [&](int64_t n) { return each ? exec_step_each(e, n) : exec_step(e, n); };
  e.groups = {&a.g};
  CHECK(step(1) == FSL_OK && step(2) == FSL_OK);  // eager, then a graph
  const int before = g_launched;
  e.groups = {&a.g, &b.g};  // a class that arrives later: its first step is captured
  g_last = cudaErrorInvalidValue;  // left by somebody else
  g_refuse = 1;
  const int rc = step(3);
  const std::string m = last_error();
  CHECK(rc == FSL_E_CUDA);
  CHECK(m.find("stage noise") != std::string::npos && m.find("refused") != std::string::npos);
  CHECK(g_launched == before);
  CHECK(step(3) == FSL_OK);
  CHECK(g_launched == before + (each ? 6 : 3));
  e.groups.clear();
  exec_destroy(e);
  return 0;
}

// An input/output step by kernels holds the buffers' device addresses: the
// same host addresses with other ones, or with copies, need a new graph.
static int io_key() {
  One a;
  CHECK(a.make(8, 3) == 0);
  Exec e;
  CHECK(exec_init(e, 0) == 0);
  e.groups = {&a.g};
  std::vector<double> host(9), map1(9), map2(9);
  auto step = [&](double* in, double* out, bool kernels) {
    a.g.io_in = a.g.io_out = host.data();
    a.g.io_bytes = sizeof(double) * 9;
    a.g.io_kernels = kernels;
    a.g.io_in_dev = in;
    a.g.io_out_dev = out;
    return exec_step(e, 1);
  };
  CHECK(exec_step(e, 1) == FSL_OK);
  const auto c0 = e.captures;
  CHECK(step(map1.data(), map1.data(), true) == FSL_OK && e.captures == c0 + 1);
  CHECK(step(map1.data(), map1.data(), true) == FSL_OK && e.captures == c0 + 1);
  CHECK(step(map2.data(), map1.data(), true) == FSL_OK && e.captures == c0 + 2);
  CHECK(step(map2.data(), map2.data(), true) == FSL_OK && e.captures == c0 + 3);
  CHECK(step(nullptr, nullptr, false) == FSL_OK && e.captures == c0 + 4);
  e.groups.clear();
  exec_destroy(e);
  return 0;
}

// Kernels may take a buffer that lies in the page-locked range as a whole
// and is aligned; everything else is left to copies.
static int mapped() {
  std::vector<double> mem(100), dev(100);
  g_pin = (char*)(mem.data() + 10);
  g_pin_dev = (char*)dev.data();
  g_pin_bytes = 50 * sizeof(double);
  for (size_t n : {1, 6, 48, 50})
    for (size_t at : {0, 2, 44, 49}) {
      double* got = mapped_doubles(mem.data() + 10 + at, n);
      CHECK(got == (at + n <= 50 ? dev.data() + at : nullptr));
    }
  CHECK(!mapped_doubles(mem.data() + 9, 1) && !mapped_doubles(mem.data() + 60, 1));
  CHECK(!mapped_doubles((char*)(mem.data() + 10) + 4, 6));
  CHECK(!mapped_doubles(mem.data() + 10, 0));
  g_pin_bytes -= 4;  // the last double is cut
  CHECK(mapped_doubles(mem.data() + 10, 49) && !mapped_doubles(mem.data() + 10, 50));
  return 0;
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "refused") return refused(false);
  if (what == "refused_each") return refused(true);
  if (what == "io_key") return io_key();
  if (what == "mapped") return mapped();
  std::printf("unknown test\n");
  return 2;
}
