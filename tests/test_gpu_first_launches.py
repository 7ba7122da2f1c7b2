"""The first launches of a process from several host threads at once.

Each kernel asks once for the shared memory it needs beyond the default, which differs with
the chunk edge and the number of worlds: threads that come first at the same time, with the
smaller sizes last, must not take away what another one has asked for.
"""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import sys, threading
    import numpy as np
    import falling_sand_engine_gb300 as fse

    fse.InitMaterials()
    fse.PushMaterials()
    order = [int(c) for c in sys.argv[1]]
    CHUNKS = (128, 16, 96, 64, 112, 32)

    def world(k):
        w = fse.World(256, 160, chunk_size=CHUNKS[k], seed=9)
        w.generate(fse.GEN_MIX, 9)
        return w

    def work(w, out, k, gate):
        gate.wait()
        for shape in (4, 0, 2):
            w.set_launch(shape)
            w.step(2)
        out[k] = (w.state(), w.particles().tobytes())

    worlds = {k: world(k) for k in order}
    out, gate = {}, threading.Barrier(len(order))
    threads = [threading.Thread(target=work, args=(worlds[k], out, k, gate)) for k in order]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in order:
        alone = {}
        work(world(k), alone, k, threading.Barrier(1))
        a, b = out[k], alone[k]
        assert a[1] == b[1] and all(np.array_equal(a[0][p], b[0][p]) for p in a[0]), k
    print("the same")
""")


@pytest.mark.parametrize("order", ["012345", "543210", "314052"])
def test_threads_launch_first_at_once(fse, order):
    r = subprocess.run([sys.executable, "-c", CHILD, order], capture_output=True, text=True, timeout=300,
                       cwd=ROOT)
    assert r.returncode == 0 and "the same" in r.stdout, r.stdout + r.stderr
