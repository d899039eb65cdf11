"""Runs with logarithms (zero modes, Fourier-accelerated gauge fixing) above 14
orders keep the order of every sum: there a logarithm amplifies rounding by
three to four per order, so that another order of summation is another field
(1e-8 of the entries of order 20 after 20 steps), and a run begun with one
engine could not be continued with the next.

The digests are SHA-256 of the links after one step, made on a B200 with the
engine's first kernels (commit 989f69b: one group of nine lanes per link,
columns and planes of components), built with CUDA 12.9.  Random start 3 of
the oracle, its Rand55(11) noise.
"""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ZM, FA = dict(zero_modes=True), dict(zero_modes=True, fa=True, alpha=0.05)
GF = dict(zero_modes=True, local_gf=True, alpha=-0.05)
OTF = dict(zero_modes=True, update="onthefly")

# L, N, engine options, thread grid, form of the grid-ordered kernels
CASES = {
    "sweep": ((4, 2, 3, 4), 15, ZM, None, "auto"),
    "fa": ((4, 4, 3, 2), 20, FA, None, "auto"),
    "fa_without_zero_modes": ((4, 4, 3, 2), 24, dict(fa=True, alpha=0.05), None, "auto"),
    "gf_team": ((4, 4, 2, 4), 16, GF, None, "team"),
    "gf_group": ((4, 4, 2, 4), 16, GF, None, "group"),
    "tlsym": ((4, 4, 2, 4), 16, dict(ZM, action="tlsym"), None, "auto"),
    "tlsym_onthefly": ((6, 3, 3, 3), 16, dict(OTF, action="tlsym"), None, "auto"),
    "float_float": ((4, 4, 2, 4), 16, dict(ZM, precision="ff"), None, "auto"),
    "onthefly": ((4, 4, 2, 4), 16, OTF, None, "auto"),
    "onthefly_team": ((4, 4, 2, 4), 20, OTF, None, "team"),
    "onthefly_group": ((4, 4, 2, 4), 16, OTF, None, "group"),
    "onthefly_segments": ((4, 4, 2, 4), 17, OTF, (2, 2, 1, 1), "auto"),
    "onthefly_many_threads": ((12, 12, 12, 12), 15, OTF, None, "auto"),
}

DIGESTS = {
    "sweep":
        "677b688586ad4d71cc5772404608ebf53b390e9e2f727998665369714d3382dd",
    "fa":
        "2ade0f51211ec8368f0bd6f6e46c366541338cedac74689689f234c1e74ae379",
    "fa_without_zero_modes":
        "55a36bf828c7c0d0954974c01c1dfad5017824afe218ada4c70a05833287f6d4",
    "gf_team":
        "b2cb5ae84f6fba8d117e3bded06207181cf7437958ab80c064f96a803bb43a10",
    "gf_group":
        "b2cb5ae84f6fba8d117e3bded06207181cf7437958ab80c064f96a803bb43a10",
    "tlsym":
        "53aa1debb765d76baa255f2a2652e976193a2c56fe3a8f7fe91f30c4b7b58f57",
    "tlsym_onthefly":
        "e9651831dc7de378f8bd005e88d03ac63269ab5da8f756d0e62efffb09a14e1e",
    "float_float":
        "dff2b18d3ede21b7d60447f1adf0dfddf353e07e6ef8878f3ff7ded1f24ee5c4",
    "onthefly":
        "3e27c618bd87ad2f4a8792be0e317ccedff815b40fe1f06635357f9b78068103",
    "onthefly_team":
        "0a07258b15b8de9673f7e8b530d5019a4f619a28fdcf1cd5679ad6b5e454fc88",
    "onthefly_group":
        "c5a2aa4e2190ed2fbd722e5ca071290d43d6463c629f5fa07e78b0b0a2cf778e",
    "onthefly_segments":
        "57fd3e6805fbeb4a8a74e26b487aab2a543446fd42dda580b349ab9038ffb72e",
    "onthefly_many_threads":
        "41f09777b85473cb3ce64a6201091dc87bc1e63317be6335ac2e68147cf6ad20",
}


def digest(P, O, name):
    L, N, kw, grid, form = CASES[name]
    o = O.Oracle(L, N)
    o.random_start(3, 0.5)
    with P.NsptEngine(L, N, **kw) as e:
        if grid:
            e.set_gf_grid(grid)
        e.set_local_gf_form(form)
        e.upload(o.links)
        e.set_noise(O.Rand55(11).gauss(o.V * 32))
        e.NsptEvolve(0.01, 1, 1)
        return hashlib.sha256(np.ascontiguousarray(e.download()).tobytes()).hexdigest()


@pytest.mark.parametrize("name", CASES)
def test_ordered_runs_keep_their_bits(engine_mod, oracle_mod, name):
    assert digest(engine_mod, oracle_mod, name) == DIGESTS[name]
