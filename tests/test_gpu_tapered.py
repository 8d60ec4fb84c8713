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


FO4 = ("S", "SMean", "k", "kMean")
FO5 = FO4 + ("momentsMean",)


@pytest.mark.parametrize("q,nx,nz,zc,npb,storage,fo,mean_bits", [
    (19, 256, 136, 32, 1, "f32", (), 32), (27, 264, 136, 32, 1, "f32", ("S", "kMean"), 32),
    (19, 256, 136, 32, 4, "f32", (), 32), (19, 264, 72, 16, 4, "f16", (), 32), (19, 256, 72, 23, 2, "f32", ("k",), 32),
    (27, 256, 72, 16, 1, "f16", FO4, 32), (27, 264, 72, 23, 1, "bf16", (), 32),
    (19, 264, 72, 16, 1, "f32", FO5, 32), (27, 256, 72, 16, 1, "f32", FO5, 64)])
def test_every_kernel_family(q, nx, nz, zc, npb, storage, fo, mean_bits):
    """Plain, 4-CTA and two-plane kernels, 16-bit storage, function objects
    with and without momentsMean."""
    assert tapers(nx, 256, nz, 32, zc)
    kw = dict(function_objects=fo, mean_bits=mean_bits, storage=storage, tile=(32, 8, 2), pop_buffers=npb)
    with Cavity(q, nx, 256, nz, 400.0, 0.05, z_chunk=zc, **kw) as a, \
            Cavity(q, nx, 256, nz, 400.0, 0.05, z_chunk=8, **kw) as b:
        for c in (a, b):
            c.init_regions()
            c.step(5)
            c.synchronize()
        for f in ("moments",) + fo:
            dtype = np.float64 if mean_bits == 64 and "Mean" in f else np.float32
            assert same_bits(a.read(f, dtype=dtype), b.read(f, dtype=dtype)), f


@pytest.mark.parametrize("q,nx,npb,storage,fo", [(19, 256, 4, "f32", ()), (27, 264, 1, "f32", FO4), (19, 256, 1, "f16", ())])
def test_monitored_steps(q, nx, npb, storage, fo):
    assert tapers(nx, 256, 72, 32, 16)
    kw = dict(function_objects=fo, storage=storage, tile=(32, 8, 2), pop_buffers=npb)
    with Cavity(q, nx, 256, 72, 400.0, 0.05, z_chunk=16, **kw) as a, \
            Cavity(q, nx, 256, 72, 400.0, 0.05, z_chunk=8, **kw) as b:
        mon = []
        for c in (a, b):
            c.init_regions()
            mon.append(c.step_monitored(6))
            c.synchronize()
        # FP64 atomics in another order
        for f in ("mass", "rho_u2"):
            np.testing.assert_allclose(mon[0][f], mon[1][f], rtol=1e-12)
        assert np.array_equal(mon[0]["nonfinite"], mon[1]["nonfinite"])
        for f in ("moments",) + fo:
            assert same_bits(a.read(f), b.read(f)), f


@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_default_shape_of_a_large_d3q19_mesh(storage):
    """Nothing named, no function objects, more than three CTAs per SM: the
    default is the 4-CTA kernel of 32-wide tiles; the bits of a named shape."""
    shape = (256, 256, 64)
    with Cavity(19, *shape, 400.0, 0.05, storage=storage) as a, \
            Cavity(19, *shape, 400.0, 0.05, storage=storage, tile=(16, 8, 2), z_chunk=8) as b:
        i = a.info()
        assert i["tile_x"] == 32 and 8 * 32 * -(-64 // i["z_chunk"]) > 3 * 148
        for c in (a, b):
            c.init_regions()
            c.step(7)
            c.synchronize()
        assert same_bits(a.read(), b.read())


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
def test_autotune_times_few_chunks_on_small_meshes(shape, most):
    """Of the chunk lengths only those are timed that may be the fastest: on a
    small mesh no more of them than powers of two and whole waves."""
    assert not tapers(*shape, 8, 16) and not tapers(*shape, 32, 16)
    with Cavity(19, *shape, 400.0, 0.05) as c:
        c.init_regions()
        assert 0 < c.autotune()["candidates"] <= most
