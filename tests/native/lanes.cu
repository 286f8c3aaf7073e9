// Host-only check of ZpLanes: the event calls are this file's own, and note who waits for whom.
#include <cstdio>
#include <string>

#include <cuda_runtime.h>

static cudaError_t test_record(cudaEvent_t e, cudaStream_t s);
static cudaError_t test_wait(cudaStream_t s, cudaEvent_t e, unsigned);
#define cudaEventRecord test_record
#define cudaStreamWaitEvent test_wait
#include "zp_core.cuh"

static std::string g_log;
static int g_fail_at = -1, g_calls = 0;
static std::string stream_name(cudaStream_t s) { return std::to_string(reinterpret_cast<size_t>(s)); }
static cudaError_t step(const std::string &what) {
  if (g_calls++ == g_fail_at) return cudaErrorInvalidValue;
  g_log += what + ' ';
  return cudaSuccess;
}
static cudaError_t test_record(cudaEvent_t e, cudaStream_t s) {
  return step("record" + std::to_string(reinterpret_cast<size_t>(e)) + "@" + stream_name(s));
}
static cudaError_t test_wait(cudaStream_t s, cudaEvent_t e, unsigned) {
  return step(stream_name(s) + "waits" + std::to_string(reinterpret_cast<size_t>(e)));
}
bool zp_lanes_enabled() { return true; }
void zp_set_cuda_error(cudaError_t, const char *) {}

// main stream 1, side streams 2 and 3, events 7 (fork), 8 and 9 (join)
static int call(const zp_plan *plan, int64_t edges, const char *script) {
  ZpLanes lanes(plan, edges, reinterpret_cast<cudaStream_t>(1));
  int rc = 0;
  for (const char *c = script; *c && !rc; c += 2) rc = c[0] == 'f' ? lanes.fork(c[1] - '0') : lanes.join(c[1] - '0');
  return rc;
}

int main(int, char **argv) {
  zp_plan plan = {};
  std::mutex lock;
  plan.lane_lock = &lock;
  plan.aux_stream[0] = reinterpret_cast<cudaStream_t>(2);
  plan.aux_stream[1] = reinterpret_cast<cudaStream_t>(3);
  plan.ev_fork = reinterpret_cast<cudaEvent_t>(7);
  plan.ev_join[0] = reinterpret_cast<cudaEvent_t>(8);
  plan.ev_join[1] = reinterpret_cast<cudaEvent_t>(9);
  g_fail_at = std::stoi(argv[3]);
  const int rc = call(&plan, std::stoll(argv[1]), argv[2]);
  std::printf("%d %d %s\n", rc, lock.try_lock() ? 1 : 0, g_log.c_str());
  return 0;
}
