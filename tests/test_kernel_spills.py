"""Registers and spills of the kernels, per instance (CPU only: nvcc cross-compiles
and ptxas reports them).

Most kernels wait on memory and are compiled for a number of resident blocks
(__launch_bounds__), which caps their registers: a build that drifts shows as
spills, or as a bound that no longer holds.  The limits are the figures that the
times in the sources were measured with."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "grass_b200", "csrc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-Xptxas", "-v"]

pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None or shutil.which("c++filt") is None,
                                reason="needs nvcc and c++filt")

# per source: {kernel (as c++filt names it): (registers, bytes of spill stores)}
LIMITS = {
    "kernels_sample.cu": {
        # 64: two blocks of 512 threads; several walkers a lane take what they need of 128
        "rw_kernel<1, 1>": (64, 0), "rw_kernel<1, 2>": (128, 0), "rw_kernel<1, 4>": (128, 128),
        "rw_csr_kernel<1>": (64, 0), "rw_csr_kernel<2>": (64, 0), "rw_csr_kernel<4>": (64, 0),
        "n2v_kernel<1>": (64, 0), "n2v_kernel<2>": (64, 0),
        "khop_kernel<1>": (64, 48), "khop_csr_kernel": (64, 24),
        # eight blocks of 256 threads
        "mrw_kernel<1>": (32, 48),
        "mrw_degree_kernel<1, 8, unsigned int>": (64, 0), "mrw_degree_kernel<1, 8, unsigned long>": (64, 0),
        "mrw_degree_kernel<1, 32, unsigned long>": (64, 0),
        # a block of 512 threads; the wide kernel a block of 1024
        "mrw_cta_kernel<1, 16>": (120, 0), "mrw_cta_kernel<1, 32>": (64, 64),
    },
    "kernels_decode.cu": {"decode_flat_kernel<1>": (64, 36)},  # 16 blocks of 64 threads
    "kernels_compact.cu": {"compact_fill_kernel<0>": (64, 0), "compact_fill_kernel<1>": (64, 0)},
    "kernels_batch.cu": {
        # four blocks of 256 threads; three with two walkers a lane, two with four (CSR: three)
        "batch_kernel<1, 1>": (64, 88), "batch_kernel<1, 2>": (80, 56), "batch_kernel<1, 4>": (128, 176),
        "batch_kernel<2, 1>": (64, 56), "batch_kernel<2, 2>": (80, 56), "batch_kernel<2, 4>": (80, 12),
        "batch_cta_kernel<1>": (64, 48), "batch_cta_kernel<2>": (64, 44),
    },
}


@pytest.mark.parametrize("src", LIMITS)
def test_registers_and_spills(tmp_path, src):
    out = subprocess.run(["nvcc", *FLAGS, "-c", os.path.join(CSRC, src), "-o", str(tmp_path / "out.o")],
                         capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
    found = re.findall(r"Function properties for (\S+)\n.*?(\d+) bytes spill stores.*?\n.*?Used (\d+) registers",
                       out.stderr)
    names = subprocess.run(["c++filt"], input="\n".join(f[0] for f in found), capture_output=True,
                           text=True).stdout.splitlines()
    seen = {n: (int(regs), int(spill)) for n, (_, spill, regs) in zip(names, found)}
    for kernel, (regs, spill) in LIMITS[src].items():
        hits = [v for n, v in seen.items() if re.search(rf"::{re.escape(kernel)}\(", n)]
        assert hits, f"no kernel {kernel}"
        for r, s in hits:
            assert r <= regs and s <= spill, f"{kernel}: {r} registers, {s} bytes spilled (at most {regs}, {spill})"
