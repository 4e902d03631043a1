"""Registers and spills of the stream and chemistry kernels as ptxas reports them for sm_103a, on the CPU:
nothing spills, 512 threads of a stream block get their registers, and the chemistry keeps the
blocks per SM that it was measured with."""
import re
import shutil
import subprocess

import pytest

from subsweep_gb300 import build


@pytest.fixture(scope="module", params=["fp64", "mixed"])
def table(request, tmp_path_factory):
    """{demangled kernel: (registers, spill store bytes)}, and the precision."""
    nvcc = shutil.which(build.NVCC)
    if nvcc is None or shutil.which("c++filt") is None:
        pytest.skip("nvcc or c++filt not available")
    src = build.CSRC / f"sweep_{request.param}.cu"
    cmd = [nvcc, *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off",
           f"-fmad={'true' if request.param == 'mixed' else 'false'}", "-Xptxas", "-v", "-c", str(src), "-o",
           str(tmp_path_factory.mktemp("ptxas") / "x.o")]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    found = {}
    for block in re.split(r"ptxas info\s*: Compiling entry function '", r.stdout + r.stderr)[1:]:
        spill = re.search(r"(\d+) bytes spill stores", block)
        regs = re.search(r"Used (\d+) registers", block)
        if spill and regs:
            found[block.split("'", 1)[0]] = (int(regs.group(1)), int(spill.group(1)))
    names = subprocess.run(["c++filt"], input="\n".join(found), capture_output=True, text=True).stdout.split("\n")
    return request.param, {dem.split("(")[0].replace("void ", ""): v for dem, v in zip(names, found.values())}


def test_stream_kernels_do_not_spill(table):
    _, kernels = table
    streams = {k: v for k, v in kernels.items() if k.startswith("swk::k_sweep_stream")}
    assert len(streams) == 17, sorted(streams)  # 4, 8, 16 warps and pairs, far words, all cells; sparse
    for name, (regs, spill) in streams.items():
        # blocks of 4 and 8 warps may have more than the 65,536 / 512 of the others
        few = re.search(r"k_sweep_stream<\w+, [48],", name)
        assert spill == 0 and regs <= (168 if few else 128), (name, regs, spill)


def test_chemistry_keeps_its_blocks_per_sm(table):
    precision, kernels = table
    (regs, spill), = [v for k, v in kernels.items() if k.startswith("swk::k_chemistry")]
    # FP64: four blocks of 128 threads; mixed: six
    assert spill == 0 and regs <= (128 if precision == "fp64" else 80), (regs, spill)
