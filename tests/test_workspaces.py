"""Workspace sizes (host arithmetic, no GPU): a kernel that reuses another's workspace fits in it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_back_transformation_fits_the_vectors_workspace(tmp_path):
    """exp, cis, functions and adjoint of one real matrix from n = 96 back-transform all 2 n columns
    (real and imaginary parts) in the workspace of the vectors when the tridiagonal splits."""
    import build_lib  # skewlinearalgebra.jl_gb300/build_lib.py

    build_lib.build()
    objs = [os.path.join(build_lib.BUILD, f) for f in sorted(os.listdir(build_lib.BUILD)) if f.endswith(".o")]
    exe = str(tmp_path / "workspaces")
    subprocess.run([build_lib._nvcc(), *build_lib.ARCH, *build_lib.FLAGS, "-I", build_lib.CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "c_caller", "workspaces.cu"), *objs], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=120).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert [r[0] for r in rows] == list(range(3, 2049))
    assert [n for n, have, need in rows if have < need] == []
