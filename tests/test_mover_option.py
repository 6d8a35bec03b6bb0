"""PIC_OPT_MOVER_CTAS_PER_SM counts CTAs of 256 threads, whatever CTA size the particle pass has: a value
asks for the same warps per SM under every kernel (host code of the library, compiled here)."""
import subprocess

from compat_io import ROOT, nvcc

PROGRAM = """
#include <cstdio>
#include "kernels.h"
int main() {
  for (int v = 0; v <= 32; ++v) std::printf("%d %d\\n", PIC_MOVER_THREADS * mover_ctas(v, 64), mover_ctas(v, 7));
}
"""


def test_option_counts_256_threads(tmp_path):
    src, exe = tmp_path / "p.cu", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run([nvcc(), "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "pic_cuda_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    rows = [tuple(map(int, r.split())) for r in subprocess.run([str(exe)], check=True, capture_output=True,
                                                              text=True).stdout.splitlines()]
    assert rows[0][1] == 7                                  # 0: as many as fit
    assert [r[0] for r in rows[1:5]] == [256, 512, 768, 1024]
    assert all(1 <= r[1] <= 7 for r in rows) and rows[32][1] == 7
