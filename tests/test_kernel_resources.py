"""Registers and spills of the collective kernels, as the assembler reports them for a few element types (no GPU needed)."""
import re
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
KERNELS = ("KAllReduceOneShot", "KAllReduceTwoShot", "KAllReduceConcurrentPlain", "KReduceScatterV", "KReduce")
TYPES = ("__nv_bfloat16", "int8_t", "double")


def _report(tmp: Path, type_: str):
    from hccl_b200.utils import build
    if not (build.CUDA_HOME / "bin" / "nvcc").exists():
        pytest.skip("no nvcc")
    src = tmp / f"{type_}.cu"
    src.write_text('#include "kernels/collectives.cuh"\nnamespace hccl { namespace {\n' + "".join(
        f"template __global__ void {k}<{type_}, false>(const DevComm *, const __grid_constant__ CollArgs, const CollArgs *);\n" for k in KERNELS) + "} }\n")
    out = subprocess.run([str(build.CUDA_HOME / "bin" / "nvcc"), "-O3", "-std=c++17", "--expt-relaxed-constexpr", *build.ARCH_FLAGS, f"-I{ROOT / 'include'}", f"-I{ROOT / 'csrc'}",
                          "-Xptxas", "-v", "-c", str(src), "-o", str(src.with_suffix(".o"))], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    return re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores.*?Used (\d+) registers", out.stderr, re.S)


def test_reducing_kernels_keep_two_ctas_per_sm_without_spilling(tmp_path):
    """512 threads at 64 registers leave room for two CTAs on an SM, which emulated ranks and concurrent operators count on. Spills of more
    than a few addresses would sit in the copy loops."""
    with ThreadPoolExecutor() as pool:
        for type_, rows in zip(TYPES, pool.map(lambda t: _report(tmp_path, t), TYPES)):
            assert len(rows) == len(KERNELS), (type_, rows)
            for name, spilled, registers in rows:
                assert int(registers) <= 64 and int(spilled) < 100, (type_, name, spilled, registers)
