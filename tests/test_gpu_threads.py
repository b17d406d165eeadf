"""Contexts of several threads on one device."""
import threading

import numpy as np
import pytest

import rg_tree
import rgpu
from refsupport import make_params
from test_gpu_level import bits_equal

pytestmark = pytest.mark.gpu


def test_line_runs_of_several_sizes_at_once(rgpu_lib):
    """rg_level_run on lines whose pieces need much and little shared memory, from a thread each: every launch is
    accepted (the opt-in to large shared memory belongs to the kernel, not to the context), same bits as alone."""
    sizes = (13, 8, 12, 7)

    def run(level, n, out, errors, start):
        try:
            g = rg_tree.build_uniform(1, level)
            u = rg_tree.sod_state(g, level, 1.4)
            ctx = rgpu.Context(make_params(1, slope_type=1, riemann="hllc"), 0)
            try:
                ctx.sync_topology(g)
                ctx.upload_state(u, u)
                start.wait(120)
                t = 0.0
                for _ in range(n):
                    t, _ = ctx.level_run(level, 1.0 / 2 ** level, 1e9, t_start=t, pressure_cap=True, max_steps=1)
                got = np.empty_like(u)
                ctx.download_state(uold=got)
                out.append((level, t, got))
            finally:
                ctx.close()
        except rgpu.RGError as e:
            errors.append(str(e))

    n, together, alone, errors = 1500, [], [], []
    start = threading.Barrier(len(sizes))
    threads = [threading.Thread(target=run, args=(s, n, together, errors, start)) for s in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for s in sizes:
        run(s, n, alone, errors, threading.Barrier(1))
    assert not errors
    for s, t, u in together:
        t1, u1 = next((b, v) for a, b, v in alone if a == s)
        assert t == t1 and bits_equal(u, u1)
