"""A cuFFT call that fails inside a call with virials leaves the context usable.

The virial's transforms run through cuFFT in the spread grid, which the
three-kernel convolution expects to be zero before every spread.  A failed plan
or transform must therefore not leave the charges already spread in it: the
solve after the failed call gives the energy and dipoles it gave before, to the
rounding of its own sums (FP64 1e-12 relative; FP32 grid 1e-6, the dipoles a few
times that).  The failures come from a stand-in for the three cuFFT entry points
(a shared library found before libcufft), so nothing fails on the GPU itself.
"""
import pathlib
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent
CUDA_LIB = "/usr/local/cuda/lib64"

# each entry point fails while its countdown reaches zero, else calls cuFFT
SHIM = textwrap.dedent("""
    #define _GNU_SOURCE
    #include <dlfcn.h>
    int shim_plans, shim_fail_plan, shim_fail_exec;  /* fail the k-th call from now (0: none) */
    static int hit(int *k) { return *k > 0 && --*k == 0; }
    int cufftPlan3d(int *p, int x, int y, int z, int t) {
      static int (*f)(int *, int, int, int, int);
      if (!f) f = dlsym(RTLD_NEXT, "cufftPlan3d");
      if (hit(&shim_fail_plan)) return 2;
      ++shim_plans;
      return f(p, x, y, z, t);
    }
    #define EXEC(name)                                      \\
      int name(int p, void *a, void *b, int d) {            \\
        static int (*f)(int, void *, void *, int);          \\
        if (!f) f = dlsym(RTLD_NEXT, #name);                \\
        return hit(&shim_fail_exec) ? 6 : f(p, a, b, d);    \\
      }
    EXEC(cufftExecC2C)
    EXEC(cufftExecZ2Z)
""")

CHILD = textwrap.dedent("""
    import ctypes, sys
    import numpy as np
    shim = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)  # before libthp and its libcufft
    plans, fail_plan, fail_exec = (ctypes.c_int.in_dll(shim, n) for n in ("shim_plans", "shim_fail_plan", "shim_fail_exec"))
    sys.path.insert(0, "tests")
    from conftest import load_package
    thp = load_package()
    from tinker_hp_b200 import lib
    precision = sys.argv[2]
    rel = 1e-12 if precision == "FP64" else 1e-6

    def refused(call):
        try:
            call()
        except lib.ThpError as e:
            assert e.status == lib.THP_E_CUDA, e
            return
        raise AssertionError("the failing cuFFT call was not reported")
""")


def run_child(tmp_path, precision, body):
    src = tmp_path / "shim.c"
    src.write_text(SHIM)
    shim = tmp_path / "libshim.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(shim), str(src), f"-L{CUDA_LIB}", "-Wl,--no-as-needed",
                    "-lcufft", f"-Wl,-rpath,{CUDA_LIB}", "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD + textwrap.dedent(body), str(shim), precision], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_solve_after_a_failed_virial_call(tmp_path, precision):
    run_child(tmp_path, precision, """
        import dataclasses
        for first, nfft in (("gradient", 20), ("empole1", 24)):  # plans are cached by grid
            ws = dataclasses.replace(thp.water.make_water_box(216, cfg=0), nfft=(nfft,) * 3)
            ctx = lib.Context(ws, precision=getattr(lib, precision))
            ref = ctx.solve()["epol"]
            mu = ctx.dipoles()[0]

            def same(what):
                got = ctx.solve()["epol"]
                assert abs(got - ref) < rel * abs(ref), (first, what, got, ref)
                assert np.abs(ctx.dipoles()[0] - mu).max() < 10 * rel * np.abs(mu).max(), (first, what)

            # the plan of the grid: refused when the virial is switched on, or
            # (made inside the call) when it first needs one
            fail_plan.value = 1
            def with_plan():
                ctx.set_virial(True)
                getattr(ctx, first)()
            refused(with_plan)
            assert fail_plan.value == 0
            same("plan")
            ctx.set_virial(True)
            getattr(ctx, first)()
            # the transforms: empole1 runs two, gradient three
            for k in range(1, 4 if first == "gradient" else 3):
                same("before")
                fail_exec.value = k
                refused(getattr(ctx, first))
                assert fail_exec.value == 0
                same(f"transform {k}")
    """)


def test_plan_is_made_when_the_virial_is_switched_on(tmp_path):
    # on a grid of the own convolution, which has none before; the calls with
    # virials, and a re-target that keeps them on, make none themselves
    run_child(tmp_path, "FP64", """
        import dataclasses
        ws = thp.water.make_water_box(216, cfg=0)
        ctx = lib.Context(ws)
        ctx.solve()
        assert plans.value == 0
        ctx.set_virial(True)
        assert plans.value == 1
        ctx.solve()
        ctx.gradient()
        ctx.empole1()
        ctx.set_virial(False)
        ctx.set_virial(True)
        assert plans.value == 1
        ctx.retarget(dataclasses.replace(ws, nfft=(24, 24, 24)))
        assert plans.value == 2
        ctx.solve()
        ctx.gradient()
        assert plans.value == 2
        # bound as the reference's virial: planned by the binding
        other = lib.Context(dataclasses.replace(ws, nfft=(30, 30, 30)))
        vir = np.zeros(9)
        fail_plan.value = 1
        assert lib.load().thp_bind_virial(other.h, lib._p(vir)) == lib.THP_E_CUDA
        assert lib.load().thp_bind_virial(other.h, lib._p(vir)) == lib.THP_OK and plans.value == 3
    """)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_batch_after_a_failed_profiled_solve(tmp_path, precision):
    # the profiled loop runs eagerly: the cuFFT class fails after both classes
    # have spread and before the other class convolves
    run_child(tmp_path, precision, """
        import dataclasses
        base = thp.water.make_water_box(216, cfg=0)
        boxes = [dataclasses.replace(base, nfft=g) for g in ((20, 24, 20), (20, 20, 20))]
        ctxs = [lib.Context(b, precision=getattr(lib, precision)) for b in boxes]
        alone = []
        for c in ctxs:
            c.solve()
            alone.append(c.dipoles()[0])
        plan = lib.Batch(ctxs)
        plan.profile(True)
        fail_exec.value = 5  # after the two convolutions of the first context's front
        refused(plan.solve)
        assert fail_exec.value == 0
        plan.profile(False)
        plan.solve()
        for c, ref in zip(ctxs, alone):
            assert np.abs(c.dipoles()[0] - ref).max() < (1e-10 if precision == "FP64" else 2e-6) * np.abs(ref).max()
    """)
