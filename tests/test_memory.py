"""Host-side parts of the engine, on the CPU: memory and error words."""
import ctypes
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def _run(tmp_path, name):
    exe = tmp_path / name
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", str(ROOT / "wipems_gb300" / "csrc"), "-I",
                        "/usr/local/cuda/include", "-o", str(exe), str(ROOT / "tests" / "glue" / f"{name}.cpp")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr


def test_device_buffer_after_a_failed_allocation(tmp_path):
    """A buffer whose allocation failed holds nothing, so the next attempt
    allocates again and no kernel gets a null pointer; a readback takes the
    scratch it can get, down to none, and then turns the axes over here; the
    threads that map its pages may fail to start at any of their allocations."""
    _run(tmp_path, "memory_harness")


def test_error_words(libs):
    """Each bounded device wait is reported as what it was."""
    from wipems_gb300 import _abi
    L = ctypes.CDLL(str(_abi.LIB_PATH))
    decode = L._ZN6wipems19engine_decode_errorEi  # wipems::engine_decode_error(int)
    for err, text in [(4, "TMA copy"), (8, "resident run"), (1, "ring overflow"), (2, "not finite")]:
        assert decode(err) != 0 and text in _abi.last_error()
    assert decode(4) == decode(8) != decode(1) and decode(0) == 0
