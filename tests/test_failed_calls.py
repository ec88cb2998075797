"""Device calls that fail on the host: the handle stays usable, nothing is left half changed.

A preloaded library stands in for the runtime's allocation and launch calls and returns their
error codes on request, so no allocation is driven to its limit and no kernel fails on the device.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
/* the runtime's own call (its library is not in the global scope: RTLD_NEXT does not see it) */
static void *real_call(const char *name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name); }
static int alloc_in = -1;   /* calls until allocations fail; -1: never */
void fake_alloc(int n) { alloc_in = n; }
int cudaMallocFromPoolAsync(void **p, size_t n, void *pool, void *stream)
{
  static int (*real)(void **, size_t, void *, void *);
  if (!real) real = (int (*)(void **, size_t, void *, void *))real_call("cudaMallocFromPoolAsync");
  if (alloc_in == 0) return 2;   /* cudaErrorMemoryAllocation */
  if (alloc_in > 0) alloc_in--;
  return real(p, n, pool, stream);
}
static int launch_in = -1, records, waits;
void fake_launch(int n) { launch_in = n; records = waits = 0; }
int fake_records(void) { return records; }
int fake_waits(void) { return waits; }
int cudaLaunchKernelExC(const void *cfg, const void *fn, void **args)
{
  static int (*real)(const void *, const void *, void **);
  if (!real) real = (int (*)(const void *, const void *, void **))real_call("cudaLaunchKernelExC");
  if (launch_in == 0) return 701;   /* cudaErrorLaunchOutOfResources */
  if (launch_in > 0) launch_in--;
  return real(cfg, fn, args);
}
int cudaEventRecord(void *event, void *stream)
{
  static int (*real)(void *, void *);
  if (!real) real = (int (*)(void *, void *))real_call("cudaEventRecord");
  records++;
  return real(event, stream);
}
int cudaStreamWaitEvent(void *stream, void *event, unsigned flags)
{
  static int (*real)(void *, void *, unsigned);
  if (!real) real = (int (*)(void *, void *, unsigned))real_call("cudaStreamWaitEvent");
  waits++;
  return real(stream, event, flags);
}
"""

PRELUDE = """
import ctypes, sys
import numpy as np
from se2dr_fork_gb300 import gpu as G, host as H, spec as S
fake = ctypes.CDLL(sys.argv[1])
"""


@pytest.fixture(scope="module")
def run_with_fake(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    src, lib = d / "fake.c", d / "libfake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)

    def run(code):
        env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
        r = subprocess.run([sys.executable, "-c", PRELUDE + code, str(lib)], cwd=ROOT, env=env, timeout=300,
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("precision", ["fp32_kahan", "fp32", "fp32_df"])
def test_failed_tile_configuration_leaves_the_handle_as_it_was(run_with_fake, precision):
    """Whatever allocation of se2gpu_set_tile_config fails, the handle goes on with the
    configuration it had: same getter, same bits."""
    run_with_fake(f"""
su = H.Setup(S.demo(19, 17, p=3, tmax=1e30).replace(nt=1000))
ref = G.Solver(su, "{precision}")
n = len(ref.tile_configs())
sol, rows, failures = G.Solver(su, "{precision}"), [], 0
for start in range(n):
    for c in range(n):
        for k in range(6):
            sol.set_tile_config(start)
            fake.fake_alloc(k)
            try:
                sol.set_tile_config(c)
            except G.GpuError as e:
                assert e.code == G.ERR_NOMEM
                failures += 1
                assert sol.tile_config == start and G.lib().se2gpu_tile_config(sol._h) == start
            fake.fake_alloc(-1)
            rows.append(sol.run(2))
want = ref.run(2 * len(rows))
assert np.array_equal(np.concatenate(rows), want)
assert all(np.array_equal(x, y) for x, y in zip(sol.fields(), ref.fields()))
assert failures >= (n - 1) * (n - 2), failures   # (two numbers may name the same tiles)
""")


@pytest.mark.parametrize("graphs", [False, True])
def test_failed_ensemble_launch_joins_its_chains(run_with_fake, graphs):
    """A block whose n-th launch fails leaves no chain running beside the ensemble's stream: each
    side chain is recorded and waited for, captured or not, and the ensemble can be set and run
    again."""
    run_with_fake(f"""
setups = [H.Setup(S.shot(7, i, size=(20 + i, 18), p=p, nt=64)) for i, p in enumerate((3, 4, 6, 3))]
def new():
    e = G.Ensemble(setups, "fp32_kahan", block=4)
    e.set_graphs({graphs})
    return e
ref = new()
want = ref.advance(8)
ens = new()
for n in range(12):   # 3 groups, one launch each per step
    fake.fake_launch(n)
    try:
        ens.advance(4, traces=False)
        raise SystemExit("the launch did not fail")
    except G.GpuError as e:
        assert e.code == -2, e
    fork, joins = 1, 2   # (the upload's event is recorded besides)
    assert fake.fake_waits() == 2 * joins and fake.fake_records() == fork + joins + 1, (fake.fake_waits(), fake.fake_records())
    fake.fake_launch(-1)
for i, su in enumerate(setups):
    ens.set_fields(i, *(np.zeros(su.ndof) for _ in range(3)))
got = ens.advance(8)
assert all(np.array_equal(x, y) for x, y in zip(got, want))
for i in range(len(setups)):
    assert all(np.array_equal(x, y) for x, y in zip(ens.fields(i), ref.fields(i)))
""")


def test_failed_ensemble_tile_configuration_is_refused_until_one_is_set(run_with_fake):
    """A tile configuration that fails for the second shot of its group leaves the group's tables
    behind: no block runs until one has been set."""
    run_with_fake("""
setups = [H.Setup(S.shot(7, i, size=(20 + i, 18), p=p, nt=64)) for i, p in enumerate((3, 4, 3))]
ref, ens = G.Ensemble(setups, "fp32_kahan", block=4), G.Ensemble(setups, "fp32_kahan", block=4)
want = [ref.advance(8), ref.advance(8)]
got = [ens.advance(8)]
for k in (0, 1):   # of the first shot, of the second
    fake.fake_alloc(k)
    try:
        ens.set_tile_config(3, 1)
        raise SystemExit("the allocation did not fail")
    except G.GpuError:
        pass
    fake.fake_alloc(-1)
    try:
        ens.advance(8)
        raise SystemExit("a block ran")
    except G.GpuError as e:
        assert e.code == -4, e   # SE2GPU_ERR_STATE
ens.set_tile_config(3, 1)
got.append(ens.advance(8))
for g, w in zip(got, want):
    assert all(np.array_equal(x, y) for x, y in zip(g, w))
""")


@pytest.mark.parametrize("call", ["traces", "fields", "norms", "checkpoint", "force", "advance", "set_fields"])
def test_failed_launch_in_an_fp64_block_leaves_whole_steps(run_with_fake, call):
    """A block whose n-th dependent launch fails has made as many whole steps as its launches began,
    whichever call comes next."""
    run_with_fake(f"""
su = H.Setup(S.demo(7, 6, p=3, tmax=1e30).replace(nt=1000))
rng = np.random.default_rng(3)
f = [rng.standard_normal(su.ndof) * s for s in (1e-6, 1e-3, 1.0)]
stf = rng.standard_normal((5, su.nsrc))
for n in range(5):   # four launches that finish a step and begin the next, and the last
    sol, ref = G.Solver(su, "fp64"), G.Solver(su, "fp64")
    for x in (sol, ref):
        x.set_fields(*f)
    fake.fake_launch(n)
    try:
        sol.advance(5, stf)
        raise SystemExit("the launch did not fail")
    except G.GpuError as e:
        assert e.code == -2, e
    fake.fake_launch(-1)
    ref.advance(n + 1, stf[:n + 1])
    sol.time, sol.step, sol._times = ref.time, ref.step, list(ref._times)
    for x in (sol, ref):
        x.got = []
        if "{call}" == "traces":
            x.got.append(x.traces())
        elif "{call}" == "fields":
            x.got += x.fields()
        elif "{call}" == "norms":
            x.got.append(x.norms())
        elif "{call}" == "force":
            x.got.append(x.assemble_linear_form(f[0]))
        elif "{call}" == "set_fields":
            x.set_fields(u=f[1])
        elif "{call}" == "checkpoint" and n == 0:   # (one row pending, none written)
            x.got.append(np.frombuffer(x.checkpoint(), dtype=np.uint8))
        x.advance(3, stf[:3])
        x.got += [x.traces(), *x.fields()]
    assert len(sol.got) == len(ref.got) and all(np.array_equal(x, y) for x, y in zip(sol.got, ref.got)), n
""")
