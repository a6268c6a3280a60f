"""Run every form of the time loops (tests/loop_shapes.py) with the library given
on the command line and print one JSON object of exact checksums, as
tests/bounds_check_run.py does for its jobs."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import numpy as np  # noqa: E402

from pseudoacousticmodeling_gb300 import _lib  # noqa: E402

_lib.load(sys.argv[1])

from tests.loop_shapes import PERSISTENT, TILES, ident  # noqa: E402
from tests.test_gpu_loop_forms import outputs, setup  # noqa: E402

out = {}
for approx, boundary, sweep, R, shape in TILES + [(a, "cerjan", "forward", 0, s) for a, s in PERSISTENT]:
    e, sz, sx, d = setup(approx, boundary, shape, nt=41)
    loop, plan = e.time_loop(len(sz), sweep)
    assert (loop, plan["R"]) == (("tiles", R) if R else ("persistent", 0)), (approx, sweep, shape, loop, plan)
    out[ident((approx, boundary, sweep, shape))] = [[float(np.float64(v).sum()), float(np.abs(np.float64(v)).sum())]
                                                    for v in outputs(e, sz, sx, d, sweep)]
    e.close()
print("CHECKSUMS " + json.dumps(out))
