"""Whole-mesh steps on grids that end in quarter chunks (z_chunks of
lbm_step.cuh): the bits of uniform chunks, in every kernel family that runs on
such grids.  Each case states its mesh and chunk and checks that they taper.
"""
import numpy as np
import pytest

from cudalbm_b200.solver import NVARS, Cavity

pytestmark = pytest.mark.gpu


def tapers(nx, ny, nz, tile_x, zc):
    """z_chunks' rule: chunks of 16 planes or more, two of them in z, and two
    waves of work (24 resident warps on each of 148 SMs)."""
    tiles = -(-nx // tile_x) * (ny // 8)
    return zc >= 16 and nz >= 2 * zc and tiles * -(-nz // zc) * (tile_x * 8 // 32) >= 2 * 148 * 24


def same_bits(a, b):
    return a.dtype == b.dtype and a.tobytes() == b.tobytes()


@pytest.mark.parametrize("q,nx,storage,fo", [(19, 256, "f32", ()), (27, 264, "f32", ("S", "kMean")), (19, 256, "f16", ())])
def test_streamed_middle_steps(q, nx, storage, fo):
    """The steps between the first and the last 16 of a streamed job run on
    the whole mesh, as lbm_step's do."""
    ny, nz, zc, n = 256, 72, 16, 37
    assert tapers(nx, ny, nz, 32, zc)
    with Cavity(q, nx, ny, nz, 400.0, 0.05, function_objects=fo, storage=storage, tile=(32, 8, 2), z_chunk=zc) as a, \
            Cavity(q, nx, ny, nz, 400.0, 0.05, function_objects=fo, storage=storage, tile=(32, 8, 2), z_chunk=8) as b:
        for c in (a, b):
            c.init_regions()
            c.step(3)
            c.synchronize()
        state = a.read()
        outs = {s: np.empty((NVARS[s],) + a.shape, np.float32) for s in ("moments",) + fo}
        a.run_streamed(state, n, outs)
        b.step(n)
        b.synchronize()
        for s, out in outs.items():
            assert same_bits(out, b.read(s)), s


@pytest.mark.parametrize("shape,most", [((64, 64, 64), 54), ((72, 40, 40), 42), ((8, 64, 64), 7)])
def test_autotune_tries_few_chunks_where_none_tapers(shape, most):
    """The lengths between the powers of two are timed on tapered grids only:
    on a small mesh a call takes no longer than powers of two and whole waves."""
    assert not tapers(*shape, 8, 16) and not tapers(*shape, 32, 16)
    with Cavity(19, *shape, 400.0, 0.05) as c:
        c.init_regions()
        assert 0 < c.autotune()["candidates"] <= most
