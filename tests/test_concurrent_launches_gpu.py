"""Host threads launch one kernel at the same time with different amounts of shared memory: a
kernel's limit belongs to the kernel, so no launch may depend on the value another one set."""
import dataclasses
import threading

import numpy as np
import pytest

from poststackmig3d_b200 import MigrationKernel, Migrator
from poststackmig3d_b200 import synth as S

from helpers import geometry_for

pytestmark = pytest.mark.gpu


def _together(jobs):
    """Runs every job (a callable) on a thread of its own, all started together; re-raises."""
    start, errors = threading.Barrier(len(jobs)), []

    def run(job):
        try:
            start.wait(timeout=60)
            job()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_threads_migrate_different_inlines_of_one_buffer():
    """The shared memory of a psm_kirchhoff_inline launch follows the output inline's place in
    its buffer (its mirror distances)."""
    n_il, n_xl, n_t = 64, 6, 40
    rng = np.random.default_rng(7)
    buf = rng.standard_normal((n_il, n_xl, n_t)).astype(np.float32)
    vel = (1800 + 400 * rng.random((n_xl, n_t))).astype(np.float32)
    il_pos = np.arange(n_il, dtype=np.int32)
    t0 = (np.arange(n_t) * 0.004).astype(np.float32)

    def migrate(cur, out):
        MigrationKernel.kirchhoff_kernel_3d_with_padding(
            buf, n_il, n_xl, n_t, vel, out, il_pos, None, cur, 0, 0.004, t0, 0.5, 25.0, 20.0,
            True)

    ref = np.empty((n_il, n_xl, n_t), dtype=np.float32)
    for c in range(n_il):
        migrate(c, ref[c])

    def job(k):
        def run():
            out = np.empty((n_xl, n_t), dtype=np.float32)
            for i in range(200):
                c = (k * 8 + i * (2 * k + 1)) % n_il
                migrate(c, out)
                assert np.array_equal(out, ref[c]), c
        return run

    _together([job(k) for k in range(8)])


@pytest.mark.parametrize("adjoint", [False, True])
def test_contexts_of_different_storage_and_size(adjoint):
    """fp32 and 16-bit traces are staged by one kernel, and an adjoint's tables follow the
    aperture: a context per thread, each with its own amount."""
    cases = []
    for precision, n_il in [("f32", 40), ("bf16", 9), ("f32", 7), ("f16", 24)]:
        W = S.random_workload(50 + n_il, n_il, 9, 60, vel_kind="linear", d_il=8.0, angle=50.0)
        cases.append((W, dataclasses.replace(geometry_for(W), precision=precision)))

    def context(W, g):
        m = Migrator(0)
        m.set_geometry(g)
        m.set_vrms(W.vrms_cube())
        m.set_traces(W.data)
        return m

    def launch(m):
        if adjoint:
            m.adjoint_async()
        else:
            m.forward_async()
        m.synchronize()

    def job(W, g):
        def run():
            with context(W, g) as m:
                m.set_image(np.ones(m.image_shape(), dtype=np.float32))
                for _ in range(300):
                    launch(m)
                if not adjoint:
                    with context(W, g) as alone:
                        assert np.array_equal(m.get_image(), alone.forward())
        return run

    _together([job(W, g) for W, g in cases])
