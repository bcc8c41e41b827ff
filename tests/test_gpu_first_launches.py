"""Grid requests that are the process's first beside a busy streamline engine.
A kernel's first launch loads its code, which waits until the device is idle, so
the engine has to have loaded every kernel of the grid path before it starts."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import time
import numpy as np
from pycpet_gb300 import core, drop_in
from pycpet_gb300.serving import Request, Server
from pycpet_gb300.synth import make_frame

srv = Server(precision="fp32c", line_capacity=100_000, charge_capacity=50_000, max_requests=64)
fr = make_frame(20000, seed=71)
srv.add_frame(0, fr["x"], fr["q"])
rng = np.random.default_rng(72)
topo = Request("topo", 0, 0.0, starts=rng.uniform(-1.5, 1.5, (60_000, 3)), n_iter=6000, step=0.001)
topo.arrival = time.perf_counter()
assert srv.submit(topo)
for _ in range(20):
    srv.step()
    time.sleep(0.005)

def mesh(k):
    g = np.linspace(-1.0, 1.0, k)
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)

grid = [Request("point_field", 0, 0.0, points=mesh(11)[:n]) for n in (1, 20, 60)]
grid += [Request(k, 0, 0.0, points=mesh(n)) for n in (5, 21, 31) for k in ("volume", "volume_esp")]
for r in grid:
    r.arrival = time.perf_counter()
    assert srv.submit(r)
t_end = time.perf_counter() + 60
while any(r.status != "done" for r in grid) and time.perf_counter() < t_end:
    srv.step()
assert all(r.status == "done" for r in grid)

class Calc:
    pass

c = Calc()
c.x, c.Q = fr["x"][:500].astype(np.float32), fr["q"][:500].astype(np.float32)
c.mesh = mesh(7).reshape(7, 7, 7, 3).astype(np.float32)
for c.precision in ("fp32c", "fp64"):
    drop_in.compute_point_field(c), drop_in.compute_box(c), drop_in.compute_box_ESP(c)
    core.field_grid(mesh(9), fr["x"][:300], fr["q"][:300], precision=c.precision)
srv.step()
assert topo.status == "running", "the grid requests waited for the streamline request"
while srv.busy() and time.perf_counter() < t_end:
    srv.step()
assert topo.status == "done"
srv.close()
"""


def test_first_grid_launches_do_not_wait_for_the_engine(gpu_lib):
    subprocess.run([sys.executable, "-c", SCRIPT], check=True, timeout=180)
