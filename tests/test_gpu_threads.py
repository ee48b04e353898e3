"""Contexts of different threads: calls that share a kernel but not its shared-memory size do not disturb each
other (the limit a kernel's launches are checked against belongs to the process, not to a context)."""
import os
import subprocess
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "hh.h"
struct job { const char *what; int n; long bad; };
static int all_ok(int rc) { return rc == HH_OK; }
/* one line of the direct DST (n 300 against 2300: 10 and 150 KB of shared memory, 2500 against 4000),
   the right-hand-side assembly (2D tiles reach 30 points, 3D tiles 17), tile input of the line solve */
static void *work(void *p) {
    struct job *j = p;
    hh_ctx *c = NULL;
    hh_plan *pl = NULL;
    double *d = NULL, *r = NULL;
    int n = j->n, three = !strcmp(j->what, "rhs3"), rhs = three || !strcmp(j->what, "rhs2"), tile = !strcmp(j->what, "tile");
    size_t e = rhs ? (size_t)(n + 2) * (n + 2) * (three ? n + 2 : 1) : tile ? (size_t)n * n : (size_t)n;
    double *host = calloc(e, 16), *k = calloc(2 * (size_t)n + 4, 8);
    int ok = all_ok(hh_ctx_create(0, NULL, &c)) && all_ok(hh_malloc(c, 16 * e, (void **)&d)) &&
             all_ok(hh_malloc(c, 16 * e, (void **)&r)) && all_ok(hh_memcpy_h2d(c, d, host, 16 * e));
    if (ok && (rhs || tile)) ok = all_ok(three ? hh_plan3d_create_helmholtz(c, n, 6, 3.0, 0.0, &pl) : hh_plan2d_create_helmholtz(c, n, 6, 3.0, 0.0, &pl));
    if (ok && tile) ok = all_ok(hh_plan_set_variant(pl, 6));
    hh_rhs2d_data d2;
    hh_rhs3d_data d3;
    memset(&d2, 0, sizeof d2);
    memset(&d3, 0, sizeof d3);
    d2.order = d3.order = 6;
    d2.hx = d2.hy = d3.hx = d3.hy = d3.hz = 1.0 / (n + 1);
    d2.f_ext = d3.f_ext = d;
    d2.k_ext = d3.k2_ext = k;
    if (!ok) { j->bad = -1; printf("%s %d: %s\n", j->what, n, hh_last_error()); return NULL; }
    for (int i = 0; i < (n > 2400 ? 300 : 2000); i++) {
        int rc = three ? hh_rhs3d(pl, &d3, r) : rhs ? hh_rhs2d(pl, &d2, r) : tile ? hh_solve_source(pl, d, d, 1) : hh_dst1_rows(c, n, 1, d, n, d, n);
        if (rc != HH_OK && j->bad++ == 0) printf("%s %d: %s\n", j->what, n, hh_last_error());
        if (i % 128 == 127) hh_ctx_synchronize(c);
    }
    if (hh_ctx_synchronize(c) != HH_OK) j->bad++;
    hh_free(c, d);
    hh_free(c, r);
    hh_ctx_destroy(c);
    return NULL;
}
int main(int argc, char **argv) {
    struct job j[2] = {{argv[1], atoi(argv[2]), 0}, {argv[3], atoi(argv[4]), 0}};
    pthread_t t[2];
    for (int i = 0; i < 2; i++) pthread_create(&t[i], NULL, work, &j[i]);
    for (int i = 0; i < 2; i++) pthread_join(t[i], NULL);
    printf("refused %ld %ld\n", j[0].bad, j[1].bad);
    return 0;
}
"""


@pytest.mark.parametrize("a,na,b,nb", [("dst", 300, "dst", 2300), ("dst", 2500, "dst", 4000), ("rhs2", 40, "rhs3", 20),
                                       ("tile", 255, "tile", 140)])
def test_two_threads_with_different_shared_memory(tmp_path, a, na, b, nb):
    src, exe, lib = tmp_path / "threads.c", str(tmp_path / "threads"), os.path.join(ROOT, "hackathon_b200")
    src.write_text(textwrap.dedent(PROGRAM))
    r = subprocess.run(["/usr/bin/gcc", "-O1", "-I", os.path.join(ROOT, "include"), str(src), "-o", exe, "-L", lib, "-lhh",
                        "-lpthread", f"-Wl,-rpath,{lib}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, a, str(na), b, str(nb)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "refused 0 0" in r.stdout, r.stdout + r.stderr
