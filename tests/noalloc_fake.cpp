// bhr_step_noalloc against a fake CUDA runtime and fake launches: what a call
// leaves behind when something fails, which no test on a device reaches
// without a fault.  Compiled and run by test_noalloc_errors.py.
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "bhr.h"
#include "bhr_host.h"
#include "bhr_internal.h"

static std::vector<std::string> calls;  // since the last forget()
static int undrained = 0;               // work enqueued and not waited for
static int resident_launches = 0, fail_resident_at = -1, fail_encode = 0;
static cudaError_t resident_error = cudaSuccess;
static unsigned long long last_seq = 0;
static double scratch[1 << 22];

static cudaError_t enqueue(const char *what) {
  calls.push_back(what);
  undrained++;
  return cudaSuccess;
}
static bool has(const std::string &w) {
  for (const auto &c : calls)
    if (c == w) return true;
  return false;
}
static int find(const std::string &w) {
  for (size_t i = 0; i < calls.size(); i++)
    if (calls[i] == w) return static_cast<int>(i);
  return -1;
}
static void forget() {
  calls.clear();
  resident_launches = 0;
}

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamGetDevice(cudaStream_t, int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = scratch, cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  if (kind == cudaMemcpyDeviceToHost) std::memset(dst, 0, n);
  return enqueue("copy");
}
cudaError_t cudaMemsetAsync(void *, int, size_t n, cudaStream_t) { return enqueue(n == sizeof(int) ? "clear flag" : "clear words"); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return undrained = 0, cudaSuccess; }
}

namespace bhr {
void set_error(const std::string &) {}
void fill_grid(const bhr_params &, double *, double *, double *, double *, double *, double *) {}
void fill_tables(const bhr_params &, double, const double *, const double *, double *, double *) {}
cudaError_t prepare_kernels() { return cudaSuccess; }
cudaError_t encode_state_maps(void *, int, int, int, CUtensorMap *, CUtensorMap *, CUtensorMap *) {
  return fail_encode ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t encode_coef_maps(double *, const double *, const double *, int, int, int, StageMaps *) { return cudaSuccess; }
cudaError_t launch_coef_tables(const double *, const double *, double *, int, int, cudaStream_t) { return enqueue("tables"); }
cudaError_t launch_closure(double *, int, int, int, cudaStream_t) { return enqueue("closure"); }
cudaError_t launch_stage(int, const StageMaps &, const StageArgs &, cudaStream_t, bool) { return enqueue("stage"); }
ResidentGeom resident_geometry(int, int, bool) { return ResidentGeom{4, 8, 4, true}; }
size_t resident_inbox_bytes(const ResidentGeom &) { return 1 << 16; }
cudaError_t launch_resident(const ResidentArgs &a, cudaStream_t) {
  if (resident_launches++ == fail_resident_at) return resident_error;
  if (a.seq <= last_seq) calls.push_back("old seq");
  last_seq = a.seq + 3ull * a.steps - 1;
  return enqueue("resident");
}
}  // namespace bhr

static int failures = 0;
static void check(bool ok, const char *what) {
  if (ok) return;
  failures++;
  std::printf("FAILED: %s\n", what);
}

static int step(bhr_params &p, int n) {
  alignas(16) static double state[4 * 256 * 32];
  forget();
  return bhr_step_noalloc(&p, state, n, nullptr);
}

int main() {
  bhr_params p{};
  p.N = 256, p.M = 32, p.Xmin = -50, p.Xmax = 50, p.mass = 1, p.a = 0.5, p.m = 2, p.dt = 0.05;
  p.precision = BHR_FP64, p.integrator = BHR_SSPRK3;

  // No room for a cooperative launch, then no tensor map: the tables and the
  // flag were enqueued, so the call waits for them before it gives the scratch up.
  fail_resident_at = 0, resident_error = cudaErrorCooperativeLaunchTooLarge, fail_encode = 1;
  check(step(p, 3) == BHR_CUDA_ERROR, "an encode failure is an error");
  check(has("tables") && undrained == 0, "a call that fails to encode its maps ends with its stream drained");
  fail_encode = 0;

  // By stage where the launch is refused; afterwards the words are cleared
  // before the next resident launch, whose numbers go on.
  check(step(p, 3) == BHR_OK && has("stage") && !has("resident"), "a refused launch goes by stage");
  fail_resident_at = -1;
  check(step(p, 3) == BHR_OK && has("resident") && !has("stage") && !has("old seq"), "resident again");
  check(find("clear words") >= 0 && find("clear words") < find("resident"), "stages are cleared out of the edge words");
  check(step(p, 3) == BHR_OK && has("resident") && !has("clear words") && !has("old seq"), "the words are kept from call to call");

  // The first launch of a long call may have set the error flag before the
  // second one failed: the next call clears it.
  check(!has("clear flag"), "the flag is not cleared after calls that ended well");
  fail_resident_at = 1, resident_error = cudaErrorLaunchFailure;
  check(step(p, 5000) == BHR_CUDA_ERROR && resident_launches == 2 && undrained == 0, "the second launch fails");
  fail_resident_at = -1;
  check(step(p, 1) == BHR_OK && find("clear flag") >= 0 && find("clear flag") < find("resident"),
        "the call after a failed one clears the flag");
  return failures != 0;
}
