"""The kernels that work in fixed point (csrc/fx.cuh) and the register-blocked transforms (csrc/fft.cuh), where they can
go wrong: both sides of every size rule, operands that the format does not hold (the kernels then fall back to FP64),
fields of a hundred orders of magnitude less, line lengths of every radix.

Tolerances.  One step is ~60 dependent FP64 roundings per number and three steps are taken: 200 x 1.1e-16 = 2e-14 of the
largest number that entered it; the bar of the other parity tests, 1e-12, leaves the oracle its own.  FP32: the same count
of 6e-8 is 1e-5.  A transform of length n makes log2 n additions per number, each of relative 1.1e-16 (FP32 6e-8) of the
largest result: below 1e-14 (5e-6) up to 2^16."""
import numpy as np
import pytest

from oracle import oracle as O
from soerenpragya3dglasma_gb300 import Lattice, build

pytestmark = pytest.mark.gpu

A, DT = (1.0, 1.1, 0.9), 0.1


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _rel(a, b):
    return np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300)


def _advance(fields, N, precision="fp64", steps=3):
    with Lattice(N, A, precision=precision) as lat:
        lat.upload_fields(fields)
        lat.step(DT, steps)
        return lat.download_fields()


# force kernel: a site over four warps up to 14592 owners nx ny (nz + 1); link kernel: a site over three blocks up to
# 12970 (FP64) and 51882 (FP32) sites
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("N", [(2, 2, 2), (5, 7, 3), (5, 1297, 2), (7, 17, 109), (16, 16, 56), (16, 16, 57),
                               (3, 8647, 2), (14, 34, 109)])
def test_step_on_both_sides_of_the_size_rules(oracle, precision, N):
    f = O.random_fields(N, 71, link_amp=0.3, e_amp=0.1, j_amp=0.05)
    if precision == "fp32":
        f = {k: v.astype(np.complex64 if np.iscomplexobj(v) else np.float32).astype(v.dtype) for k, v in f.items()}
    ref = O.copy_fields(f)
    oracle.update(ref, N, A, DT, 3)
    out = _advance(f, N, precision)
    for k in O.FIELD_NAMES:
        assert _rel(out[k], ref[k]) < (1e-12 if precision == "fp64" else 1e-5), k


def _out_of_range(kind, N):
    f = O.random_fields(N, 72, link_amp=0.3, e_amp=0.1, j_amp=0.05)
    rng = np.random.default_rng(5)
    if kind == "scaled_links":  # entries above one
        f["U"][rng.random(f["U"].shape[:3]) < 0.15] *= 1.5
    elif kind == "short_links":
        f["U"][rng.random(f["U"].shape[:3]) < 0.15] *= 0.5
    elif kind == "strong_fields":  # |dt E| of one and more
        f["E"][rng.random(f["E"].shape[:3]) < 0.3] *= 300.0
    elif kind == "drift":  # nothing to fall back for, but not unitary either
        f["U"] *= 1 + 1e-6
    f["UOld"] = f["U"].copy()
    for k in O.FIELD_NAMES:
        O.sync_ghosts(f[k])
    return f


@pytest.mark.parametrize("N", [(6, 5, 8), (16, 16, 80)])
def test_strong_fields_fall_back(oracle, N):
    f = _out_of_range("strong_fields", N)
    ref = O.copy_fields(f)
    oracle.update(ref, N, A, DT, 1)
    out = _advance(f, N, steps=1)
    for k in O.FIELD_NAMES:
        assert _rel(out[k], ref[k]) < 1e-12, k


# Links that are not unitary: every method of the step has its own answer then (plaquettes are rotated where the reference
# multiplies staples), so the force in fixed point is compared with the same force in double-float arithmetic, 1e-13 as on
# unitary links, and the energies, which are products of the links as they are, with the oracle.
@pytest.mark.parametrize("kind", ["scaled_links", "short_links", "drift"])
@pytest.mark.parametrize("N", [(6, 5, 8), (16, 16, 80)])
def test_links_off_the_group_fall_back(oracle, kind, N):
    f = _out_of_range(kind, N)
    out = {}
    for mode in ("native", "double_float"):
        with Lattice(N, A) as lat:
            lat.upload_fields(f)
            if mode == "native":
                assert np.allclose(lat.bulk(), oracle.bulk(f, N, A), rtol=1e-12, atol=1e-10)
                assert np.allclose(lat.unitarity(), oracle.unitarity(f, N), rtol=1e-9)
            lat.set_step_method("plaquette")
            lat.fp64_arithmetic = mode
            lat.step(DT, 1)
            out[mode] = lat.download_fields()
    for k in O.FIELD_NAMES:
        assert _rel(out["native"][k], out["double_float"][k]) < 1e-13, k


@pytest.mark.parametrize("size", [1e-30, 1e-110, 1e-200])
def test_dilute_slices_keep_their_digits(oracle, size):
    """Slices whose fields are `size` of the others', as in the tails of a nucleus: relative accuracy slice by slice."""
    N = (4, 5, 24)
    f = O.random_fields(N, 73, link_amp=0.2, e_amp=0.1, j_amp=0.05)
    far = slice(10, N[2] + 2)
    f["U"][far] = O.new_fields(N)["U"][far]
    f["UOld"] = f["U"].copy()
    for k in ("E", "Jp", "Jm", "JpStat", "JmStat"):
        f[k][far] *= size
    ref = O.copy_fields(f)
    oracle.update(ref, N, A, DT, 2)
    out = _advance(f, N, steps=2)
    for z in range(16, N[2] + 1):  # out of reach of the strong half
        for k in ("E", "Jp", "Jm", "JpStat", "JmStat"):
            assert _rel(out[k][z], ref[k][z]) < 1e-12, (k, z)
        assert 0 < np.max(np.abs(out["U"][z].imag)) < size
        assert _rel(out["U"][z].imag, ref["U"][z].imag) < 1e-12, z


# E^2 is summed in fixed point for fields between 2^-100 and 2^50
@pytest.mark.parametrize("amp,e_amp", [(0.02, 1e-2), (0.3, 1e-33), (0.3, 1e17)])
@pytest.mark.parametrize("N", [(3, 2, 2), (9, 7, 33)])
def test_fp32_energy_and_unitarity_of_the_stored_fields(oracle, amp, e_amp, N):
    """FP32 lattices are measured in fixed point: against the oracle on the numbers that the lattice holds.  A plaquette half
    is a product in FP32 (6e-8 of its size)."""
    f = O.random_fields(N, 74, link_amp=amp, e_amp=e_amp, j_amp=0.02)
    with Lattice(N, A, precision="fp32") as lat:
        lat.upload_fields(f)
        got, uni = lat.bulk(), lat.unitarity()
        held = lat.download_fields()
    want = oracle.bulk(held, N, A)
    for k in (0, 1, 2):
        assert abs(got[k] - want[k]) <= 1e-12 * abs(want[k]), k
    for k in (3, 4, 5):
        assert abs(got[k] - want[k]) <= 1e-6 * abs(want[k]), k
    assert np.allclose(uni, oracle.unitarity(held, N), rtol=1e-3, atol=1e-15)


# links as FP32 leaves them (deviations of 1e-7, 1e-16 / 1e-7 known in FP64), exact ones, and ones that fall back
@pytest.mark.parametrize("amp,scale", [(0.3, 1.0), (0.0, 1.0), (0.3, 0.5), (0.3, 1.5)])
@pytest.mark.parametrize("N", [(2, 2, 2), (9, 7, 33)])
def test_fp32_unitarity(oracle, amp, scale, N):
    f = O.random_fields(N, 79, link_amp=amp)
    f["U"][::2] *= scale
    with Lattice(N, A, precision="fp32") as lat:
        lat.upload("U", f["U"])
        got = lat.unitarity()
        held = lat.download("U")
    assert np.allclose(got, oracle.unitarity({"U": held}, N), rtol=1e-8, atol=0)


LENGTHS = [2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 25, 27, 32, 45, 60, 64, 81, 96, 125, 128, 160, 240, 243, 256, 360, 486, 512, 625, 720,
           1024, 2048, 3000, 4096, 6561, 8192, 7, 14, 22, 49, 1001]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_transform_lengths(n, axis):
    N = [3, 5, 2]
    N[axis] = n
    rng = np.random.default_rng(n)
    shape = (8, N[2], N[1], N[0])
    x = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    x32 = x.astype(np.complex64)
    with Lattice(tuple(N)) as lat:
        got = [lat.fft3d(x), lat.fft3d(x, inverse=True), lat.fft3d_f32(x32), lat.fft3d_f32(x32, inverse=True)]
    x32 = x32.astype(np.complex128)
    sites, axes = x[0].size, (1, 2, 3)
    want = [np.fft.fftn(x, axes=axes), np.fft.ifftn(x, axes=axes) * sites, np.fft.fftn(x32, axes=axes),
            np.fft.ifftn(x32, axes=axes) * sites]
    for i, (g, w) in enumerate(zip(got, want)):
        assert _rel(g, w) < (1e-14 if i < 2 else 5e-6), i


# the acceleration step along z in one pass (lengths 2^a 3^b 5^c) and as three kernels (others), on tiles of sixteen lines
# and ragged ones
@pytest.mark.parametrize("project", [False, True])
@pytest.mark.parametrize("N", [(4, 4, 16), (5, 3, 30), (6, 6, 9), (3, 6, 64), (4, 4, 14), (2, 3, 200)])
def test_gauge_sweeps_on_ragged_lattices(oracle, N, project):
    rng = np.random.default_rng(9)
    f = O.random_fields(N, 75, link_amp=0.02, e_amp=0.1)
    G = O.identity_gauge(N)
    st, olog, UG, EG = oracle.coulomb_fix(f, G, N, (1.0, 1.0, 1.0), 0.5, 3, flags=O.GF_PROJECT_ZERO_MODE if project else 0)
    assert st == 0
    with Lattice(N) as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        log = lat.coulomb_fix(0.5, 3, project_zero_mode=project)
        assert np.allclose(log, olog, rtol=1e-10, atol=1e-13)
        assert np.max(np.abs(lat.download("G") - G)) < 1e-11
        assert np.max(np.abs(lat.download("UG") - UG)) < 1e-11
        assert np.max(np.abs(lat.download("EG") - EG)) < 1e-11


# G leaves the FP32 sweeps by the expansion about SU(3), or, further than 2^-17 from it, by Newton's iteration.  Both are
# exact to rounding (1e-4 squared twice); the products of an entry and of the determinant, and the few FP64 sweeps that may
# follow, add some ten roundings each: 1e-14.
@pytest.mark.parametrize("scale", [1.0, 1 + 1e-4])
@pytest.mark.parametrize("N,iters", [((3, 2, 4), 2), ((9, 7, 11), 40)])
def test_mixed_sweeps_leave_su3(scale, N, iters):
    f = O.random_fields(N, 80, link_amp=0.2)
    with Lattice(N) as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        lat.upload("G", scale * O.identity_gauge(N))
        lat.coulomb_fix(0.08, iters, open_z=True, mixed=True)
        G = O.links_as_matrices(lat.download("G"))[1:-1]
    assert np.max(np.abs(G @ np.swapaxes(G.conj(), -1, -2) - np.eye(3))) < 1e-14
    assert np.max(np.abs(np.linalg.det(G) - 1)) < 1e-14


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("N", [(2, 2, 2), (5, 3, 7), (33, 4, 3)])
def test_device_buffers_give_the_same_bytes(precision, N):
    torch = pytest.importorskip("torch")
    f = O.random_fields(N, 76)
    with Lattice(N, precision=precision) as a, Lattice(N, precision=precision) as b:
        for k in ("U", "E", "Jp"):
            dev = torch.from_numpy(f[k].view(np.float64).copy()).cuda()
            torch.cuda.synchronize()
            a.upload_device(k, dev.data_ptr())
            b.upload(k, f[k])
            out = torch.empty_like(dev)
            a.download_device(k, out.data_ptr())
            a.synchronize()
            assert np.array_equal(out.cpu().numpy(), b.download(k).view(np.float64)), k


@pytest.mark.parametrize("e_amp", [1e-4, 0.5, 6.0, 30.0])
def test_adjoint_across_field_strengths(e_amp):
    """The exponential's pull-back as a series (|q| below one) and in closed form: the derivative along a random direction
    against central differences.  eps = 1e-6 of the field: truncation 1e-12, rounding 1e-16 / 1e-6 = 1e-10 of the
    objective."""
    N, steps = (4, 5, 10), 2
    f = O.random_fields(N, 77, link_amp=0.25, e_amp=e_amp, j_amp=0.05)
    d = e_amp * np.random.default_rng(3).standard_normal(f["E"].shape)
    O.sync_ghosts(d)

    def value(E):
        with Lattice(N, A) as lat:
            lat.upload_fields(dict(f, E=E))
            lat.step(DT, steps, save_uold=False)
            return lat.objective(2, 8, Lattice.ENERGY)

    with Lattice(N, A) as lat:
        lat.upload_fields(f)
        L, g = lat.adjoint(DT, steps, 2, 8, Lattice.ENERGY, checkpoint_every=1)
    eps = 1e-6
    fd = (value(f["E"] + eps * d) - value(f["E"] - eps * d)) / (2 * eps)
    ad = float(np.sum(g["E"][1:-1] * d[1:-1]))
    assert abs(fd - ad) <= 1e-5 * max(abs(fd), 1e-3 * abs(L))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_adjoint_is_zero_beyond_reach(precision):
    """No step carries a cotangent further than two slices: it is exactly zero beyond, not the rounding of a neighbour's."""
    N, steps = (4, 4, 30), 2
    f = O.random_fields(N, 78, link_amp=0.25, e_amp=0.3, j_amp=0.05)
    with Lattice(N, A, precision=precision) as lat:
        lat.upload_fields(f)
        _, g = lat.adjoint(DT, steps, 14, 16, Lattice.ENERGY, checkpoint_every=1)
    for k, v in g.items():
        assert np.all(v[1:8] == 0) and np.all(v[24:-1] == 0), k
        assert np.any(v[15] != 0), k
