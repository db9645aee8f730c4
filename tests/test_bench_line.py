"""bench.py's reference arm on CPU: one JSON line in the contract's shape,
its config built by the same function as the GPU arm's line (so the two
lines describe the same workload), and an end-to-end figure that moves no
bytes between host and device."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    sys.path.insert(0, ROOT)
    import importlib.util
    spec = importlib.util.spec_from_file_location("bench_mod", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    return bench


def test_profiles_are_stamped_with_every_kernel_header():
    """A capture taken before any header of the element loop changed is not
    reported as current."""
    bench = _bench()
    from alya_sma_b200 import build as B
    csrc = {os.path.basename(p) for p in bench.KERNEL_SOURCES if "/csrc/" in p}
    assert set(B.HEADERS) | {"sma_capi.cu"} <= csrc
    assert all(os.path.exists(os.path.join(ROOT, p)) for p in bench.KERNEL_SOURCES)


def test_line_names_the_kernel_that_runs():
    bench = _bench()
    solo, lanes = {"block": 64, "variant": "plain"}, {"block": 32, "variant": "plain"}
    assert bench.element_kernel(solo, "fp32", 2_000_000) == "k_element_solo"
    assert bench.element_kernel(lanes, "fp64", 640) == "k_element"
    assert bench.element_kernel(solo, "surrogate", 2_000_000) == "k_element_sur"
    assert bench.element_kernel(lanes, "fp32", 2_000_000, block=32) == "k_element_solo"
    assert bench.element_kernel(solo, "fp32", 2_000_000, block=64, variant="plain") == "k_element"
    assert bench.element_kernel(solo, "fp32", 2_000_000, block=64, scatter="color") == "k_element"
    assert bench.element_kernel({"block": 256, "variant": "pipe"}, "fp32", 2_000_000) == "k_element_pipe"


def test_reference_arm_line_on_a_small_cylinder():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--div", "8",
                          "--steps", "2", "--warmup", "1"], capture_output=True, text=True, cwd=ROOT,
                         timeout=600)
    assert out.returncode == 0, out.stderr
    lines = [l for l in out.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1, out.stdout
    d = json.loads(lines[0])
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
              "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert k in d, k
    assert d["impl"] == "reference" and d["value"] > 0 and d["higher_is_better"] is True
    assert d["e2e"]["h2d_bytes_per_step"] == 0 and d["e2e"]["d2h_bytes_per_step"] == 0
    assert d["cpu_baseline"]["value"] == d["value"] and d["cpu_baseline"]["cores"] >= 1
    bench = _bench()
    args = bench.parse(["--div", "8"])
    args.partition = False
    prob = bench.build_problem(args.workload, args.div)
    want = bench.arm_config(args, 1, prob.nelem, prob.npoin, prob.nelem * 8, bench.working_set(prob, args.precision))
    assert d["config"] == want, (d["config"], want)
    assert "fits the 126 MB L2" in d["config"]["l2"]
