"""Launch shapes are tuned per kernel: runs that take different kernels have different keys.

Otherwise a shape tuned in one field is applied in another; two particles per thread,
tuned in an affine field, took dipole and uniform runs off their own kernels.
"""
import subprocess
from pathlib import Path


def test_kernels_have_their_own_variant(tp, tmp_path):
    root = Path(__file__).resolve().parent
    csrc = Path(tp._abi.LIB_PATH).parent / "csrc"
    exe = tmp_path / "kernel_variants"
    nvcc = next(p for p in ("/usr/local/cuda/bin/nvcc", "nvcc") if p == "nvcc" or Path(p).exists())
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr", f"-I{csrc}",
                    str(root / "kernel_variants.cu"), "-o", str(exe)], check=True, capture_output=True)
    rows = [[int(x) for x in line.split()] for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    names = ["dipole", "uniform", "affine", "b_only", "b_uniform_e", "eb_large", "eb_small", "cubic", "coop"]
    fp64, fp32c = (dict(zip(names, r)) for r in rows)
    assert fp64.pop("coop") == fp64["cubic"]               # FP32C only
    assert len(set(fp64.values())) == len(fp64)
    assert fp32c.pop("b_only") == fp32c["b_uniform_e"]     # float64 only
    assert len(set(fp32c.values())) == len(fp32c)
