"""Table Vrms of short traces and small tables, on both sides of the rule that gives a sample a
thread of its own instead of a place in a work item: the host provider's bits, exact hits
included."""
import numpy as np
import pytest

from poststackmig3d_b200 import Migrator, plan_geometry
from poststackmig3d_b200 import host as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_t", [1, 2, 20, 63, 64, 126, 127, 129, 200])
@pytest.mark.parametrize("n_il,n_xl,n_points", [(1, 1, 3), (7, 9, 1), (5, 13, 66), (40, 31, 5)])
def test_table_vrms_of_short_traces(tmp_path, n_il, n_xl, n_t, n_points):
    rng = np.random.default_rng(n_t * 100 + n_points)
    il = np.arange(3, 3 + 2 * n_il, 2, dtype=np.int32)
    xl = np.arange(10, 10 + n_xl, dtype=np.int32)
    pts = [(int(rng.choice(il)), int(rng.choice(xl)), float(rng.integers(0, n_t) * 0.004 +
                                                            rng.choice([0.0, 1e-6, 0.001])),
            float(np.float32(rng.uniform(1500, 3500)))) for _ in range(n_points)]
    pts[-1] = (int(il[-1]), int(xl[-1]), (n_t - 1) * 0.004, 2222.0)  # hits the last sample
    t = tmp_path / "t.txt"
    t.write_text("".join(f"{a} {b} {c!r} {d!r}\n" for a, b, c, d in pts))
    host = H.velocity_cube(str(t), il, xl, n_t, 0.004)
    g = plan_geometry(n_il, n_xl, n_t, 0.004, 25.0, 25.0, 30.0, 3000.0, il_labels=il,
                      xl_labels=xl)
    with Migrator(0) as m:
        m.set_geometry(g)
        m.set_vrms_table(pts, il, xl)
        got = m.get_vrms()
    assert np.array_equal(got, host)
