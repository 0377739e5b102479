"""The bounds-checked library on the kernels that the default configuration picks
from the grid (test_gpu_bounds.py runs the explicit tile heights): short FP64
tiles with two lanes a face, 7-row FP32 and learned tiles, the marching tile of
the single solve and of the batch with no, every and some faces listed, and the
device state copies.  Its guard record must stay empty and its results equal the
release library's (the bounds of test_gpu_bounds.py)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_bounds import FLAG_FRACTION, FP32_REL_TOL, PKG, _cfg

# (testcase, nx, ny, seed, scheme, rk, precision): TILE_I 0
SMALL = [
    (4, 17, 40, 3, 1, 2, 0), (3, 37, 29, 0, 0, 1, 0), (1, 100, 100, 0, 2, 2, 0), (5, 6, 6, 2, 3, 0, 0),
    (4, 17, 40, 3, 1, 2, 1), (3, 100, 33, 0, 0, 1, 1), (0, 6, 6, 0, 2, 2, 1), (2, 15, 97, 0, 3, 0, 1),
    (5, 17, 40, 3, 1, 2, 2), (3, 100, 33, 0, 0, 1, 2),
]
# more than 912 tiles of 16 x 32, in odd numbers of rows and columns
LARGE = [(5, 701, 707, 5, 1, 2, 2), (3, 17, 14700, 0, 0, 1, 2), (5, 14620, 33, 5, 2, 2, 2)]
MANY = [(5, 700, 450, 5), (0, 6, 6, 0), (3, 17, 33, 0), (5, 305, 641, 6)]
NETWORKS = ("none", "all", "some")


def _network(kind):
    """Flags no node, every node (a constant logit far from the threshold) or, as
    the initial weights do, some."""
    import wenofd

    if kind == "some":
        return wenofd.mlp_init(11)
    p = np.zeros(wenofd.MLP_PARAMS, np.float32)
    p[-1] = 4.0 if kind == "all" else -4.0
    return p


def run_all(path):
    import torch

    import wenofd

    out = {}

    def copies(s, name):
        """The state through a caller's dense device array, guarded by a value on each side."""
        n = 4 * s.nx * s.ny
        x = torch.full((n + 2,), -7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        lib = wenofd.lib()
        assert lib.wenofd_get_state_device(s.handle, x.data_ptr() + 8) == wenofd.OK
        assert lib.wenofd_set_state_device(s.handle, x.data_ptr() + 8) == wenofd.OK
        s.info()  # waits for the solver's stream
        assert x[0] == -7.0 and x[-1] == -7.0
        out[name] = s.get_state()
        assert np.array_equal(x[1:-1].cpu().numpy(), out[name].ravel())

    for k, c in enumerate(SMALL + LARGE):
        for net in NETWORKS if c[6] == wenofd.LEARNED else ("",):
            with wenofd.Solver(_cfg(*c, 0)) as s:
                s.initialize()
                if net:
                    s.set_indicator(_network(net), 0.5)
                assert s.advance(max_steps=3) == 3
                copies(s, f"{c[6]}_{k}_{net}_state")
                if net:
                    out[f"{c[6]}_{k}_{net}_flags"] = s.routing_flags()
    for precision, members, tile in ((0, [(4, 16, 12, 3), (3, 37, 29, 0)], None), (2, MANY, (16, 1))):
        for net in NETWORKS if precision == wenofd.LEARNED else ("",):
            for rk in (1, 2):
                solvers = [wenofd.Solver(_cfg(tc, nx, ny, sd, 1, rk, precision, 0)) for tc, nx, ny, sd in members]
                try:
                    for s in solvers:
                        s.initialize()
                        if net:
                            s.set_indicator(_network(net), 0.5)
                    with wenofd.Batch(solvers) as b:
                        assert b.tile() == tile if tile else b.tile()[1] == 2
                        b.advance(3)
                    for m, s in enumerate(solvers):
                        copies(s, f"{precision}_batch{rk}{m}_{net}_state")
                        if net:
                            out[f"{precision}_batch{rk}{m}_{net}_flags"] = s.routing_flags()
                finally:
                    for s in solvers:
                        s.close()
    report = wenofd.bounds_report(reset=False)
    out["guard"] = np.array([report["count"], report["line"], report["index"], report["extent"]])
    out["guard_where"] = np.array(report["where"])
    np.savez(path, **out)


@pytest.mark.gpu
def test_default_tiles_under_the_guards(tmp_path):
    sys.path.insert(0, PKG)
    import build

    got = {}
    for name, library in (("checked", build.build_checked()), ("release", None)):
        env = dict(os.environ)
        env.pop("WENOFD_LIBRARY", None)
        if library:
            env["WENOFD_LIBRARY"] = library
        path = str(tmp_path / (name + ".npz"))
        r = subprocess.run([sys.executable, os.path.abspath(__file__), path], env=env, capture_output=True, text=True,
                           timeout=900)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
        got[name] = np.load(path)
    a, b = got["checked"], got["release"]
    assert a["guard"][0] == 0, f"{a['guard']} at {a['guard_where']}"
    assert b["guard"][0] == -1
    for k in b.files:
        if k.startswith("guard"):
            continue
        x, y = a[k], b[k]
        if k.endswith("_some_state"):  # a node whose flag differs takes the other flux
            assert np.all(np.isfinite(x)), k
        elif k.endswith("flags"):
            assert np.count_nonzero(x != y) <= FLAG_FRACTION * x.size, k
        elif k.startswith("0_"):
            assert np.array_equal(x, y), k
        else:
            assert np.max(np.abs(x - y)) <= FP32_REL_TOL * np.max(np.abs(y)), k


if __name__ == "__main__":
    sys.path.insert(0, os.path.join(PKG, "python"))
    run_all(sys.argv[1])
