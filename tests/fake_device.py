"""Builds tests/host/fake_device.cpp with the library's host sources and runs
a test's scenario on it, in a process of its own (the package loads one library
per process)."""
import os
import pathlib
import shutil
import subprocess
import sys

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "cenote_b200" / "csrc"


def build(out: pathlib.Path) -> pathlib.Path:
    """The library's C++ files over a device that computes nothing. Kernels and
    CUDA calls that fake_device.cpp does not define succeed and do nothing."""
    from cenote_b200 import build as b

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = pathlib.Path(nvcc).resolve().parent.parent / "include"
    b.OUT.mkdir(parents=True, exist_ok=True)
    tables = b._tables_blob().parent
    sources = [CSRC / s for s in b.CPP_SOURCES] + [ROOT / "tests" / "host" / "fake_device.cpp"]
    objects = [out / (s.name + ".o") for s in sources]
    flags = ["g++", "-O1", "-std=c++17", "-fPIC", "-ffp-contract=off", f"-I{CSRC}", f"-I{include}", f"-I{tables}"]
    jobs = [subprocess.Popen([*flags, "-c", str(s), "-o", str(o)]) for s, o in zip(sources, objects)]
    assert [j.wait() for j in jobs] == [0] * len(jobs)

    def symbols(flag):
        text = subprocess.run(["nm", flag, *map(str, objects)], check=True, capture_output=True, text=True).stdout
        return {line.split()[-1] for line in text.splitlines() if line.strip() and not line.endswith(":")}

    missing = symbols("--undefined-only") - symbols("--defined-only")
    stubs = out / "stubs.c"
    stubs.write_text("".join(f"long {s}(void) {{ return 0; }}\n" for s in sorted(missing)
                             if s.startswith(("_ZN2cn", "cuda"))))
    lib = out / "libfake_device.so"
    subprocess.run(["gcc", "-w", "-fno-builtin", "-fPIC", "-c", str(stubs), "-o", str(out / "stubs.o")], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", str(lib), *map(str, objects),
                    str(out / "stubs.o"), "-lpthread"], check=True)
    return lib


def run(lib: pathlib.Path, test_file: str, scenario: str) -> None:
    r = subprocess.run([sys.executable, test_file, str(lib), scenario], capture_output=True, text=True, timeout=120,
                       env={**os.environ, "PYTHONPATH": f"{ROOT}:{ROOT / 'tests'}"})
    assert r.returncode == 0, r.stdout + r.stderr


def main(scenarios: dict) -> None:
    """The scenario process: the package on the fake library, its controls passed in."""
    import ctypes

    import cenote_b200

    cenote_b200.LIB_PATH = pathlib.Path(sys.argv[1])
    lib = cenote_b200.library()
    for name in ("live_bytes", "meminfo_calls", "bad_launches", "windowed_walks", "window_free_shadows",
                 "open_windows", "late_stages", "waves", "sorts", "largest_wave"):
        getattr(lib, "fake_" + name).restype = ctypes.c_uint64
    lib.fake_limit.argtypes = lib.fake_refuse_above.argtypes = [ctypes.c_uint64]
    lib.fake_stream.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
    lib.fake_stream.restype = ctypes.c_void_p
    lib.fake_clock_ms.restype = ctypes.c_double
    scenarios[sys.argv[2]](lib)
