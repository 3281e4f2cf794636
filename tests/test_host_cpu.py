"""Error paths of the host layer that need no GPU: its sources compiled into a small program without a context."""
import glob
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


OPTIN = r"""
#include "smem_optin.h"
#include <chrono>
#include <stdio.h>
#include <thread>
int main() {
    // two threads with a context each on one device: one of them asks first and takes its time in the driver
    for (int first = 0; first < 2; first++) {
        SmemOptIn opt;
        std::atomic<size_t> set{0};
        size_t seen[2];
        const size_t want[2] = { 100, 150 };
        auto ask = [&](int i) {
            opt.raise(0, want[i], [&](size_t n) { std::this_thread::sleep_for(std::chrono::milliseconds(i == first ? 200 : 1)); set = n; return 0; });
            seen[i] = set;                            // what a launch of this thread would meet
        };
        std::thread a(ask, first);
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
        std::thread b(ask, 1 - first);
        a.join(); b.join();
        if (seen[0] < 100 || seen[1] < 150 || set != 150) { printf("%zu %zu %zu\n", seen[0], seen[1], set.load()); return 1; }
        if (opt.raise(0, 160, [](size_t) { return 7; }) != 7) return 2;               // a refusal is passed on and not remembered
        if (opt.raise(0, 155, [&](size_t n) { set = n; return 0; }) != 0 || set != 155) return 3;
        if (opt.raise(1, 10, [&](size_t n) { set = n; return 0; }) != 0 || set != 10) return 4;     // another device has its own
    }
    return 0;
}
"""


def test_shared_memory_opt_in_only_grows(tmp_path):
    src, exe = tmp_path / "optin.cpp", tmp_path / "optin"
    src.write_text(OPTIN)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{LIB}/csrc", "-o", str(exe), str(src), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)


def test_every_opt_in_goes_through_it():
    """A kernel is opted in to the size of a call only through the growing opt-in; two others ask once for a fixed size."""
    for path in glob.glob(os.path.join(LIB, "csrc", "*.cu")):
        code = open(path).read()
        if "cudaFuncAttributeMaxDynamicSharedMemorySize" in code:
            assert "std::call_once" in code and "(int)smem)" not in code and "(int)csmem)" not in code, path


UPLOAD = r"""
#include "ib_b200_internal.h"
#include <stdlib.h>
#include <string.h>
static char* area; static int copies, fail_at = -1, in_flight;
static struct { void* dst; const void* src; size_t n; } queued[4096];
static int fake_stage(int slot, size_t bytes, void** h, void** d) { (void)slot; area = realloc(area, bytes ? bytes : 1); *h = area; *d = NULL; return 0; }
static int fake_sync(ibcu_ctx* c) { (void)c; for (int i = 0; i < in_flight; i++) memcpy(queued[i].dst, queued[i].src, queued[i].n); in_flight = 0; return 0; }
static int fake_h2d(ibcu_ctx* c, void* dst, const void* src, size_t n) {       /* leaves the staging area as late as the device may */
    (void)c;
    if (copies++ == fail_at) return -2;
    queued[in_flight].dst = dst; queued[in_flight].src = src; queued[in_flight++].n = n;
    return 0;
}
#define ib_b200_stage fake_stage
#define ibcu_sync_spin fake_sync
#define ibcu_memcpy_h2d fake_h2d
#include "ib_b200_pq.c"
#include <stdio.h>
int main(void) {
    const size_t sizes[] = { 1, KM_PIECE - 1, KM_PIECE, 5 * KM_PIECE + 7, KM_STAGE, KM_STAGE + 3, 40u << 20 };
    for (int s = 0; s < 7; s++)
        for (int rep = 0; rep < 5; rep++) {
            const size_t n = sizes[s];
            char *src = malloc(n), *dst = calloc(n, 1);
            for (size_t i = 0; i < n; i++) src[i] = (char)(i * 2654435761u >> 13) + rep;
            if (km_upload(dst, src, n)) return 1;
            fake_sync(NULL);
            if (memcmp(src, dst, n)) { printf("size %zu differs\n", n); return 2; }
            copies = 0; fail_at = (int)(n / KM_PIECE / 2);                     /* a transfer that fails ends the call, helpers and all */
            if (km_upload(dst, src, n) != -2) return 3;
            in_flight = 0; fail_at = -1;
            free(src); free(dst);
        }
    return 0;
}
"""


def test_kmeans_upload_in_pieces(tmp_path):
    """Pieces copied by several threads into a staging area that is used more than once: every byte arrives, and a transfer that fails
    leaves no thread behind."""
    src, exe = tmp_path / "up.c", tmp_path / "up"
    src.write_text(UPLOAD)
    subprocess.run(["gcc", "-std=gnu11", "-O2", "-w", f"-I{ROOT}/include", f"-I{LIB}/host", "-o", str(exe), str(src), f"{LIB}/host/ib_b200_table.c",
                    f"-L{LIB}", "-libcu", f"-Wl,-rpath,{LIB}", "-lm", "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)


WAIT = r"""
#include "wait_clock.h"
#include <stdio.h>
static int looks(unsigned long long ns, unsigned long long at) { WaitClock c; int n = 1; while (!c.spent(at)) { at += ns; if (++n > 100000000) return -1; } return n; }
int main() {
    const unsigned long long start[] = { 1, 1ull << 40, (1ull << 52) - 3000000000ull, ~0ull - 1000000000ull };   // the short reading wraps, the long one too
    for (unsigned long long at : start) {
        const int n = looks(1000000, at);                    // a look every millisecond: some two seconds
        if (n < 2000 || n > 2300) { printf("%d looks of a millisecond\n", n); return 1; }
        if (looks(10000000000ull, at) != 10) return 2;       // looks ten seconds apart end too
        WaitClock c;
        for (int i = 0; i < 7; i++) {                        // stopped for a minute seven times, a few microseconds of waiting between
            if (c.spent(at)) return 3;
            at += 60000000000ull;
            if (c.spent(at)) return 4;
            at += 5000;
        }
    }
    return 0;
}
"""


def test_a_stopped_kernel_does_not_run_out_of_time(tmp_path):
    """A wait that comes back after the GPU served somebody else goes on; every wait ends."""
    src, exe = tmp_path / "wait.cpp", tmp_path / "wait"
    src.write_text(WAIT)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{LIB}/csrc", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)
    code = open(os.path.join(LIB, "csrc", "tc_common.cuh")).read()
    assert "clock.spent(now)" in code


HELPERS = r"""
#define _GNU_SOURCE
#include <pthread.h>
#include <sched.h>
#include <signal.h>
#include <stdlib.h>
#include <string.h>
static int started, open_signals;
static int counted_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    sigset_t now;
    pthread_sigmask(SIG_SETMASK, NULL, &now);                /* what the new thread inherits */
    started++;
    if (!sigismember(&now, SIGUSR1) || !sigismember(&now, SIGTERM)) open_signals++;
    return pthread_create(t, a, f, arg);
}
#define pthread_create counted_create
#include "ib_b200_internal.h"
static char* area;
static int fake_stage(int slot, size_t bytes, void** h, void** d) { (void)slot; area = realloc(area, bytes); *h = area; *d = NULL; return 0; }
static int fake_sync(ibcu_ctx* c) { (void)c; return 0; }
static int fake_h2d(ibcu_ctx* c, void* dst, const void* src, size_t n) { (void)c; memcpy(dst, src, n); return 0; }
#define ib_b200_stage fake_stage
#define ibcu_sync_spin fake_sync
#define ibcu_memcpy_h2d fake_h2d
#include "ib_b200_pq.c"
#include <stdio.h>
int main(void) {
    const size_t n = 3 * KM_SHARED + 5;
    char *src = malloc(n), *dst = malloc(n);
    for (size_t i = 0; i < n; i++) src[i] = (char)(i * 31);
    cpu_set_t all, one;
    if (sched_getaffinity(0, sizeof all, &all)) return 1;
    const int cores = CPU_COUNT(&all);
    sigset_t now;
    if (km_upload(dst, src, n) || memcmp(src, dst, n)) return 2;
    if (started != (cores - 1 < KM_HELPERS ? cores - 1 : KM_HELPERS)) { printf("%d helpers on %d cores\n", started, cores); return 3; }
    if (open_signals) { printf("%d helpers take signals\n", open_signals); return 4; }
    pthread_sigmask(SIG_SETMASK, NULL, &now);
    if (sigismember(&now, SIGUSR1)) return 5;                /* the caller's own mask is back */
    int c = 0;
    while (!CPU_ISSET(c, &all)) c++;
    CPU_ZERO(&one); CPU_SET(c, &one);
    if (sched_setaffinity(0, sizeof one, &one)) return 6;
    started = 0;
    memset(dst, 0, n);
    if (km_upload(dst, src, n) || memcmp(src, dst, n)) return 7;
    if (started) { printf("%d helpers beside the caller on its only core\n", started); return 8; }
    return 0;
}
"""


def test_copy_helpers_take_no_signals_and_no_core_that_is_not_there(tmp_path):
    src, exe = tmp_path / "helpers.c", tmp_path / "helpers"
    src.write_text(HELPERS)
    subprocess.run(["gcc", "-std=gnu11", "-O2", "-w", f"-I{ROOT}/include", f"-I{LIB}/host", "-o", str(exe), str(src), f"{LIB}/host/ib_b200_table.c",
                    f"-L{LIB}", "-libcu", f"-Wl,-rpath,{LIB}", "-lm", "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)


STEP = r"""
#include "ibcu.h"
#include <stdio.h>
static int products, silu, known;
static int fake_linear(ibcu_ctx* c, const ibcu_linear_t* t, int n, const float* x, int N, int B, int bits, const ibcu_prologue_t* p) {
    (void)c; (void)t; (void)n; (void)x; (void)N; (void)B; (void)bits;
    if (p) { silu += p->op == IBCU_PRO_SILU_MUL; known += p->op == IBCU_PRO_KNOWN_MAX; }
    return 0;
}
static int fake_product(ibcu_ctx* c, float* o, const float* g, const float* u, int n, int B, float* a, int parts) { (void)c; (void)o; (void)g; (void)u; (void)n; (void)B; (void)a; (void)parts; products++; return 0; }
#define ibcu_linear_ex fake_linear
#define ibcu_silu_mul_amax fake_product
#define ibcu_embed_rows(...) 0
#define ibcu_attention_decode_at(...) 0
#define ibcu_attention_decode(...) 0
#include "ib_b200_forward.c"
int main(void) {
    layer y = { 0 };
    ib_b200_model m = { 0 };
    m.world = 1; m.L = &y; m.c.n_layers = 1; m.c.hidden = 4096;
    const int wide[] = { 11008, IBCU_PREPARED_COLUMNS, IBCU_PREPARED_COLUMNS + 32, 28672 };
    for (int w = 0; w < 4; w++)
        for (int B = 1; B <= 32; B++) {
            const int want = B >= 4 && w < 2;                /* the product where the digits are made, or in a launch with its maximum */
            products = silu = known = 0;
            m.c.inter = wide[w];
            if (issue(&m, 0, B, 1) || silu != want || known != !want || products != !want) { printf("%d wide, %d positions: %d %d %d\n", wide[w], B, silu, known, products); return 1; }
        }
    return 0;
}
"""


def test_where_a_step_forms_the_product_of_the_mlp(tmp_path):
    """Rows that one pass of the preparation does not hold keep the launch of their own: many blocks form the product there, where the preparation would
    have one block per position."""
    src, exe = tmp_path / "step.c", tmp_path / "step"
    src.write_text(STEP)
    subprocess.run(["gcc", "-std=gnu11", "-O2", "-w", f"-I{ROOT}/include", f"-I{LIB}/host", "-o", str(exe), str(src), f"-L{LIB}", "-libcu", f"-Wl,-rpath,{LIB}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)
