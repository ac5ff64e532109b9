"""The serving worker when a device call fails, on the CPU: sb_serve.cpp is compiled against stand-ins for the grouped
engine and the CUDA runtime, whose calls fail on request. An engine's failure has to end that engine's requests with its
error (not with the energies of spins that missed steps), leave the other engine's alone, and not outlast its cause."""
import os
import subprocess

import pytest

from annealing_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "sb_serve.cpp"

// what fails, by replica tile (0: nothing)
static std::atomic<int> fail_tables{0}, fail_steps{0}, expire{0}, steps_without_tables{0};
static std::atomic<int> recorded{0};  // the runtime's last error

// ---- CUDA: device memory is host memory ----
extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 1; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaFreeHost(void *) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return (cudaError_t)recorded.exchange(0); }
const char *cudaGetErrorString(cudaError_t) { return "launch refused"; }
sb_status sb_create(sb_ctx **c, const sb_device_opts *) { *c = nullptr; return SB_ERR_NO_DEVICE; }
sb_status sb_destroy(sb_ctx *) { return SB_OK; }
sb_status sb_set_wait_limit(sb_ctx *, int64_t) { return SB_OK; }
sb_status sb_solve(sb_ctx *, const sb_problem *, const sb_params *, sb_result *) { return SB_ERR_NO_DEVICE; }
const char *sb_last_error(sb_ctx *) { return ""; }
int64_t sb_plan_footprint(const sb_problem *, const sb_params *) { return 1; }
}
std::string sbh::device_status_text(uint32_t) { return "a bounded wait gave up"; }
sb_status sbh::energy_i64(const sb_problem *, const int8_t *, int64_t *out, int) { *out = -7; return SB_OK; }

// ---- the grouped engine ----
namespace sbk {
bool grouped_supports(const sb_problem *, const sb_params *) { return true; }
int64_t grouped_instance_bytes(int, int, int, int, int) { return 1; }
Grouped::~Grouped() {}
bool Grouped::wave_takes(int, int, int, int, int) { return true; }
int Grouped::steps_per_launch(const GHost &, int) { return 1; }
sb_status Grouped::prepare(GHost &g, const sb_problem *p, const sb_params *prm, uint64_t, int tag, int, cudaStream_t, Staging &,
                           std::string &, int) {
  g.tag = tag;
  g.n = g.xp = p->n;
  g.R = prm->replicas;
  g.x = (float *)calloc((size_t)g.R * g.xp, sizeof(float));
  g.energy = (double *)calloc(g.R, sizeof(double));
  return SB_OK;
}
void Grouped::release(GHost &g, cudaStream_t) {
  free(g.x);
  free(g.energy);
}
void Grouped::attach(GHost &g, int) {
  insts.push_back(g);
  dirty = true;
}
void Grouped::remove(int i) {
  release(insts[i], nullptr);
  insts.erase(insts.begin() + i);
  dirty = true;
}
sb_status Grouped::sync_tables(std::string &err) {
  if (!dirty) return SB_OK;
  if (!d_status) d_status = (uint32_t *)calloc(1, sizeof(uint32_t));
  n_items = (int)insts.size();
  if (fail_tables == nr) {
    err = "no room";
    return SB_ERR_OOM;
  }
  dirty = false;
  return SB_OK;
}
cudaError_t Grouped::run_steps(int, int, bool) {
  if (dirty) ++steps_without_tables;
  if (fail_steps == nr) {
    recorded = (int)cudaErrorLaunchOutOfResources;
    return cudaErrorLaunchOutOfResources;
  }
  if (recorded != 0) return (cudaError_t)recorded.load();  // a launch looks at the last error
  if (expire == nr) {
    *d_status |= kErrWaitTimeout;
    expire = 0;
  }
  return cudaSuccess;
}
cudaError_t Grouped::energy_pass_for(const std::vector<int> &idx, int) {
  for (int i : idx)
    for (int r = 0; r < insts[i].R; ++r) insts[i].energy[r] = -7.0;
  return cudaSuccess;
}
}  // namespace sbk

static sbs::Server *server;
static uint64_t submit(int R, int steps) {
  static float J[16] = {0};
  static sb_problem p;
  p.n = 4;
  p.J = J;
  p.integer_valued = 1;
  sb_params prm;
  memset(&prm, 0, sizeof(prm));
  prm.replicas = R;
  prm.steps = steps;
  uint64_t t = 0;
  sbs::server_submit(server, &p, &prm, &t);
  return t;
}
static void poll(const char *what, uint64_t t) {
  sb_result r;
  memset(&r, 0, sizeof(r));
  std::string err;
  const sb_status s = sbs::server_poll(server, t, &r, 20000, err);
  printf("%s %d %d %s\n", what, (int)s, r.energy_check_ok, err.c_str());
}

int main() {
  std::string err;
  sbs::server_create(&server, 0, 1 << 20, 64, err);
  for (auto *flag : {&fail_steps, &fail_tables})
    for (int tile : {32, 64}) {
      *flag = tile;
      const uint64_t a = submit(32, 300), b = submit(64, 300), c = submit(48, 700);
      poll("r32", a);
      poll("r64", b);
      poll("r48", c);
      *flag = 0;
      const uint64_t d = submit(32, 100), e = submit(64, 100);
      poll("r32", d);
      poll("r64", e);
    }
  for (int tile : {32, 64}) {
    expire = tile;
    const uint64_t a = submit(32, 300), b = submit(64, 300);
    poll("r32", a);
    poll("r64", b);
    const uint64_t d = submit(32, 100), e = submit(64, 100);
    poll("r32", d);
    poll("r64", e);
  }
  printf("stepped without tables %d\n", steps_without_tables.load());
  sbs::server_destroy(server);
}
"""

def _status(name):
    for line in open(os.path.join(ROOT, "include", "sb.h")):
        f = line.split()
        if len(f) > 2 and f[0] == name and f[1] == "=":
            return int(f[2].rstrip(","))
    raise AssertionError(name)


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    d = tmp_path_factory.mktemp("serve")
    src, exe = d / "serve.cpp", d / "serve"
    src.write_text(PROGRAM)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build._nvcc()))), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "annealing_gb300", "csrc"), "-I", cuda, str(src), "-o", str(exe), "-lpthread"], check=True)
    out = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, timeout=120)
    assert out.returncode == 0
    return out.stdout.splitlines()


def test_each_engine_ends_its_own_requests(lines):
    cuda, oom = _status("SB_ERR_CUDA"), _status("SB_ERR_OOM")
    want = []
    for failing, text in ((cuda, "steps: launch refused"), (oom, "instance tables: no room")):
        bad, good = f"{failing} 0 {text}", "0 1 "
        want += [f"r32 {bad}", f"r64 {good}", f"r48 {good}", f"r32 {good}", f"r64 {good}"]   # tile 32 fails
        want += [f"r32 {good}", f"r64 {bad}", f"r48 {bad}", f"r32 {good}", f"r64 {good}"]    # tile 64
    bad, good = f"{_status('SB_ERR_TIMEOUT')} 0 a bounded wait gave up", "0 1 "
    want += [f"r32 {bad}", f"r64 {good}", f"r32 {good}", f"r64 {good}"]
    want += [f"r32 {good}", f"r64 {bad}", f"r32 {good}", f"r64 {good}"]
    want += ["stepped without tables 0"]
    assert lines == want
