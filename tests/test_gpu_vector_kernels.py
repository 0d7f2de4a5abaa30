"""The PCG's vector kernels where their paths part: grids on either side of the chunk count up to
which the x/r pass takes a CTA's whole chunk at once, instances with and without GHOST tiles side by
side (the p.Ap sum of its own launch or of the last CTA), pure-Neumann and open instances in one
batch (the mean of r with the x/r pass), partial chunks.  Each instance gives the bits of its solve
alone, and of the unfused V-cycle's iteration, whose sums are the chunked ones throughout."""
from __future__ import annotations

import numpy as np
import pytest

from cirrus_b200 import DeviceGrid, GMGSolver

pytestmark = pytest.mark.gpu


def rhs(b, seed):
    g = DeviceGrid(b.topology)
    rng = np.random.default_rng(seed)
    for a in range(3):
        g.set_channel(6 + a, b.velocity[a] * rng.uniform(0.5, 2.0))
    g.projection_rhs()
    r = g.get_channel(1)
    g.close()
    return r


def solve(topos, bs, pure, **kw):
    g = DeviceGrid(topos)
    for i, b in enumerate(bs):
        g.set_channel_instance(i, 1, b)
    res = GMGSolver().solve_batch(g, pure_neumann=pure, max_iters=20, **kw)
    out = [g.get_channel_instance(i, 0).view(np.uint32) for i in range(len(bs))]
    g.close()
    return res, out


@pytest.mark.parametrize("names", [
    ["uniform32_small"],                                              # 8 chunks, no GHOST tiles
    ["uniform32_small", "sphere64_small"],                            # one instance without GHOST tiles
    ["sphere64_small", "sphere64_neumann_small", "ring64_small"],     # open and closed boxes
    ["sphere256_neumann"],                                            # 470 chunks
    ["sphere256_neumann", "ring64_small", "sphere256"],               # over the line: 956 chunks
])
def test_batches_across_the_paths(names, built_cache):
    bs = [built_cache(n) for n in names]
    b = [rhs(x, i) for i, x in enumerate(bs)]
    pure = [x.workload.pure_neumann for x in bs]
    res, out = solve([x.topology for x in bs], b, pure)
    for i, x in enumerate(bs):
        one, bits = solve([x.topology], [b[i]], [pure[i]])
        assert res[i] == one[0] and np.array_equal(out[i], bits[0]), names[i]


@pytest.mark.parametrize("name", ["uniform32_small", "sphere64_small", "sphere64_neumann_small", "ring64_small", "sphere256_neumann"])
def test_fused_and_unfused_iterations_agree(name, built_cache, monkeypatch):
    b = built_cache(name)
    r, pure = rhs(b, 1), [b.workload.pure_neumann]
    a = solve([b.topology], [r], pure)
    monkeypatch.setenv("CIRRUS_VCYCLE", "generic")
    e = solve([b.topology], [r], pure)
    assert a[0][0][0] == e[0][0][0] and abs(a[0][0][1] - e[0][0][1]) <= 1e-12 * e[0][0][1]
    assert np.array_equal(a[1][0], e[1][0])
