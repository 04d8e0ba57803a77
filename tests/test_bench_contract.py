"""bench.py's reference arm runs without a GPU (the FP64 oracle on the host
cores): one JSON line with the keys of the benchmark line, alone and under
torchrun with two ranks (rank 0 prints, the other exits 0 without work)."""
import json
import os
import socket
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KEYS = {"metric", "value", "unit", "impl", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
        "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"}


def _lines(out):
    return [json.loads(x) for x in out.splitlines() if x.startswith("{")]


def _check(line, n_gpus):
    assert KEYS <= set(line), KEYS - set(line)
    assert line["impl"] == "reference" and line["n_gpus"] == n_gpus
    assert line["metric"] == "particle-steps/s" and line["higher_is_better"] is True and line["value"] > 0
    assert line["config"]["workload"] == "wcsph_dam_break_128k"
    cb = line["cpu_baseline"]
    assert cb["kind"] in ("port", "reference") and cb["cores"] >= 1 and cb["value"] == line["value"]
    e = line["e2e"]
    assert e["value"] == line["value"] and e["h2d_bytes_per_step"] == 0 and e["d2h_bytes_per_step"] == 0


def test_reference_arm_line():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"],
                       cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = _lines(r.stdout)
    assert len(lines) == 1
    _check(lines[0], 1)


def test_reference_arm_under_torchrun():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", "2",
           "--master-addr", "127.0.0.1", "--master-port", str(port), "bench.py", "--impl", "reference",
           "--gpus", "2", "--steps", "1", "--warmup", "1"]
    r = subprocess.run(cmd, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = _lines(r.stdout)
    assert len(lines) == 1
    _check(lines[0], 2)


def test_counts_of_other_kernels_are_not_reported(tmp_path):
    """The captured counts belong to the code they were captured from: a change
    of the kernels drops them, one of their comments does not."""
    sys.path.insert(0, ROOT)
    import bench

    for p in bench.CAPTURED_SOURCES:
        (tmp_path / p).parent.mkdir(parents=True, exist_ok=True)
        (tmp_path / p).write_text("// one\n__global__ void k(int* a) { /* two */ a[0] = 1; }\n")
    (tmp_path / "profiles").mkdir()
    js = tmp_path / "profiles" / "traffic.json"
    assert bench.captured_counts(root=str(tmp_path)) == {}
    sha = {p: bench.code_hash(str(tmp_path / p)) for p in bench.CAPTURED_SOURCES}
    js.write_text(json.dumps({"k_sph_accel_bytes_per_launch": 5, "code_sha256": sha}))
    assert bench.captured_counts(root=str(tmp_path))["k_sph_accel_bytes_per_launch"] == 5
    src = tmp_path / bench.CAPTURED_SOURCES[0]
    src.write_text("__global__ void k(int* a)\n{ a[0] = 1;  // three\n}\n")
    assert bench.captured_counts(root=str(tmp_path))["k_sph_accel_bytes_per_launch"] == 5
    src.write_text("__global__ void k(int* a) { a[0] = 2; }")
    assert bench.captured_counts(root=str(tmp_path)) == {}
    js.write_text(json.dumps({"k_sph_accel_bytes_per_launch": 5}))
    assert bench.captured_counts(root=str(tmp_path)) == {}
