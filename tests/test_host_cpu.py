"""Error paths of the host layer that need no GPU: its sources compiled into a small program without a context."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "libinferbit_b200")

KMEANS = r"""
#include "ib_b200_pq.c"
#include <stdio.h>
int main(void) {
    float X[64] = {0}, centers[8] = {0};
    km_bufs b;
    memset(&b, 0xAA, sizeof b);                      /* what a stack may hold */
    if (km_begin(&b, X, 8, 8, 1, centers) == 0) return 1;      /* no context: the first allocation fails */
    const void* v[] = { b.X, b.C, b.idx, b.dist, b.sums, b.counts, b.inertia, b.shift };
    for (int i = 0; i < 8; i++) if (v[i]) { printf("field %d is set\n", i); return 2; }
    return 0;
}
"""


def test_kmeans_buffers_are_empty_when_a_step_fails(tmp_path):
    src, exe = tmp_path / "km.c", tmp_path / "km"
    src.write_text(KMEANS)
    subprocess.run(["gcc", "-std=gnu11", "-O2", "-w", f"-I{ROOT}/include", f"-I{LIB}/host", "-o", str(exe), str(src), f"{LIB}/host/ib_b200_table.c",
                    f"-L{LIB}", "-libcu", f"-Wl,-rpath,{LIB}", "-lm", "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)
