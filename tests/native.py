"""Host-side pieces of the library compiled into a test's own program."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vrad_gb300" / "csrc"


def run(tmp_path, program, sources=()):
    """Compiles `program` (C++) with `sources` of the library and returns what it prints."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    from vrad_gb300 import build

    main, exe = tmp_path / "main.cpp", tmp_path / "main"
    main.write_text(program)
    cuda = build._cuda_home(build._nvcc())
    cmd = [cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), "-I", str(cuda / "include"), str(main),
           *[str(CSRC / s) for s in sources], "-o", str(exe), "-L", str(cuda / "lib64"), "-lcudart", "-lpthread", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300,
                       env={"LD_LIBRARY_PATH": str(cuda / "lib64")})
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    return r.stdout
