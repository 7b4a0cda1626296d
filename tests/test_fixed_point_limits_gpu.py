"""The limits of the fixed-point kernels (csrc/fx.cuh): numbers that the format holds differently or not at all, which have
to come out as FP64 gives them.

Tolerances.  The kernels and the oracle each make some tens of FP64 roundings of 1.1e-16 per site: 1e-12 of the largest
number of a slice, the bar of the other parity tests.  What is stored in FP32 adds its own rounding, 6e-8."""
import numpy as np
import pytest

from oracle import oracle as O
from soerenpragya3dglasma_gb300 import GlasmaError, Lattice, build

pytestmark = pytest.mark.gpu

A = (1.0, 1.1, 0.9)


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _rotated(V, e):
    """2 tr(t^a V (t.e) V^dagger)."""
    return O.algebra_from_herm(V @ O.herm_from_algebra(e) @ np.swapaxes(V.conj(), -1, -2))


def _random_gauge(N, seed):
    """A random SU(3) matrix per site in the layout of G, [.., j, i], ghost slices synced."""
    G = O.random_fields(N, seed, link_amp=0.8)["U"][..., 0, :, :].copy()
    O.sync_ghosts(G)
    return G


# ---- FP32 lattices: zeros and subnormal numbers
@pytest.mark.parametrize("links", ["identity", "random"])
def test_fp32_zero_fields_measure_exactly_zero(links):
    N = (5, 4, 6)
    with Lattice(N, A, precision="fp32") as lat:
        if links == "random":
            lat.upload("U", O.random_fields(N, 90, link_amp=0.3)["U"])
            lat.upload("G", _random_gauge(N, 91))
        lat.upload("E", O.zero_efield(N))
        worst, mean, profile = lat.gauss(profile=True)
        assert worst == 0 and mean == 0 and not profile.any()
        assert not lat.emt_map().any()  # UOld is the identity
        lat.coulomb_fix(0.08, 0)
        assert not lat.download("EG").any()


@pytest.mark.parametrize("size", [1e-22, 1e-33, 1e-36, 1e-40, 1e-43])
def test_fp32_dilute_slices(oracle, size):
    """Slices of E at `size`, half of their components zero, beside slices of order one."""
    N = (5, 4, 12)
    f = O.random_fields(N, 92, link_amp=0.3, e_amp=0.1, j_amp=0.0)
    f["UOld"] = O.identity_links(N)
    f["E"][6:] *= 10 * size
    f["E"][6:][np.random.default_rng(1).random(f["E"][6:].shape) < 0.5] = 0.0
    O.sync_ghosts(f["E"])
    G = _random_gauge(N, 93)
    with Lattice(N, A, precision="fp32") as lat:
        lat.upload_fields(f)
        held = lat.download_fields()
        profile, emt = lat.gauss(profile=True)[2], lat.emt_map()
        lat.upload("G", G)
        g = O.links_as_matrices(lat.download("G"))
        lat.coulomb_fix(0.08, 0)
        EG = lat.download("EG")
    want_p, want_t = oracle.gauss(held, N, A, profile=True)[2], oracle.emt_map(held, N, A)
    want_e = _rotated(g[..., None, :, :], held["E"])
    for z in range(N[2]):
        assert abs(profile[z] - want_p[z]) <= 1e-12 * want_p[z], z
        assert np.max(np.abs(emt[z] - want_t[z])) <= 1e-12 * want_t[z, 0], z
        # stored in FP32: half an ulp of the largest component, or of the subnormal numbers (1.4e-45)
        d, top = np.abs(EG[z + 1] - want_e[z + 1]), np.max(np.abs(want_e[z + 1]))
        assert np.max(d) <= 6e-8 * top + 0.8e-45, z


# ---- links far from SU(3): what the fixed-point sums cannot hold goes through FP64
@pytest.mark.parametrize("u", [0.6, 0.74, 0.78, 0.9, 1.02, 1.2])
@pytest.mark.parametrize("N", [(2, 2, 2), (9, 7, 33)])
def test_fp32_norms_of_links_off_the_group(N, u):
    """The same matrix on every link, all entries u + iu: the products of a plaquette's halves are equal, and the FP32 bulk
    energy is -2 (n(a) + n(b) + n(c) + n(d)) per plaquette, n = ||link||^2 - 3."""
    U = np.full((N[2] + 2, N[1], N[0], 3, 3, 3), u + 1j * u)
    with Lattice(N, A, precision="fp32") as lat:
        lat.upload("U", U)
        magnetic = lat.bulk()[3:6]
    n = 18 * float(np.float32(u)) ** 2 - 3
    assert np.allclose(magnetic, -8 * n * N[0] * N[1] * N[2], rtol=1e-12, atol=0)


# A matrix that is far from unitary although every entry is below 1.03, and an algebra vector whose rotation by it adds up to
# more than the format's 8 in the eighth component: the columns (or rows) of V lie along eigenvectors of t.e.
ALONG = 0.99 * np.array([-1.0, 0, 0, -1, 0, -1, 0, 0])  # 2 t.e has eigenvalues -1.98 along (1,1,1) and 0.99 across


def _far_matrix(columns):
    return 1.02 * (1 + 1j) * np.array(columns, dtype=np.complex128).T


ROTATES_BEYOND = _far_matrix([(1, -1, 0), (1, -1, 0), (1, 1, 1)])
PAIR_BEYOND = _far_matrix([(1, 1, 1), (1, 1, 1), (1, -1, 0)])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("sign", [1, -1])
def test_transports_by_links_off_the_group(oracle, precision, sign):
    N = (4, 3, 5)
    f = O.new_fields(N)
    f["U"][...] = ROTATES_BEYOND.T  # [.., j, i]
    f["E"][...] = sign * ALONG
    with Lattice(N, A, precision=precision) as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        held = lat.download_fields()
        got, emt = lat.gauss(profile=True), lat.emt_map()
        G = np.broadcast_to(ROTATES_BEYOND.conj(), O.identity_gauge(N).shape).copy()  # G = V^dagger, stored [.., j, i]
        lat.upload("G", G)
        g = O.links_as_matrices(lat.download("G"))
        lat.coulomb_fix(0.08, 0)
        EG = lat.download("EG")
    want = oracle.gauss(held, N, A, profile=True)
    for k in range(3):
        assert np.allclose(got[k], want[k], rtol=1e-12, atol=0), k
    want = oracle.emt_map(held, N, A)
    assert np.max(np.abs(emt - want)) <= 1e-12 * np.max(np.abs(want))
    want = _rotated(g[..., None, :, :], held["E"])
    assert np.max(np.abs(EG - want)[1:-1]) <= (1e-12 if precision == "fp64" else 1e-7) * np.max(np.abs(want))


@pytest.mark.parametrize("N", [(4, 3, 8), (16, 16, 80)])  # a site over four warps, or in one thread
@pytest.mark.parametrize("which", ["Jp", "Jm"])
def test_currents_through_links_off_the_group(which, N):
    """JStat after one step at the slice above a layer of such z links: its rotation is by that link, its plaquettes are not.
    The pair of rotations takes the last diagonal entry from the trace, as the FP64 kernels do."""
    dt, z0 = 0.1, 3
    f = O.random_fields(N, 94, link_amp=0.3, e_amp=0.1, j_amp=0.0)
    f["U"][z0 + 1, ..., 2, :, :] = PAIR_BEYOND.T
    f[which][...] = ALONG
    with Lattice(N, A) as lat:
        lat.upload_fields(f)
        lat.set_step_method("plaquette")
        lat.step(dt, 1)
        got = lat.download(which + "Stat")[z0 + 2]
    C = PAIR_BEYOND.conj().T @ O.herm_from_algebra(ALONG) @ PAIR_BEYOND
    C[2, 2] = -(C[0, 0] + C[1, 1])
    want = (-1 if which == "Jp" else 1) * dt / A[2] * (ALONG - O.algebra_from_herm(C))
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


# ---- Coulomb gauge fixing: weak fields keep their digits, transformations off the group go through FP64
def _weak_links(N, seed, size):
    """1 + i q - q^2 / 2 with q of `size`: the entries themselves, where an eigenvector form would round at 1e-16."""
    q = size * O.herm_from_algebra(np.random.default_rng(seed).standard_normal((N[2] + 2, N[1], N[0], 3, 8)))
    return O.matrices_to_links(np.eye(3) + 1j * q - 0.5 * q @ q)


def _synced(F):
    O.sync_ghosts(F)
    return F


@pytest.mark.parametrize("size", [1e-4, 1e-10, 1e-20, 1e-60])
@pytest.mark.parametrize("fft_fp32", [False, True])
def test_gauge_fixing_of_weak_fields(oracle, size, fft_fp32):
    """Deviations relative to the fields' size.  The log's steps are 3 - tr X ~ size^2, which FP64 forms cannot hold."""
    N = (6, 5, 8)
    f = O.random_fields(N, 95, e_amp=0.1)
    f["U"] = _synced(_weak_links(N, 96, size))
    G = O.identity_gauge(N)
    iters = 1 if fft_fp32 else 3  # FP32 transforms round the step at 6e-8
    st, olog, UG, _ = oracle.coulomb_fix(f, G, N, (1.0, 1.0, 1.0), 0.08, iters, tol=1e-300,
                                         flags=O.GF_PROJECT_ZERO_MODE | O.GF_OPEN_Z)
    assert st == 0
    with Lattice(N) as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        log = lat.coulomb_fix(0.08, iters, tol=1e-300, project_zero_mode=True, open_z=True, fft_fp32=fft_fp32)
        got = lat.download("UG")
    assert np.allclose(log[:, 1:3], olog[:, 1:3], rtol=1e-12, atol=0)
    assert np.allclose(log[:, 5:], olog[:, 5:], rtol=1e-12, atol=0)
    if not fft_fp32:
        off = ~np.eye(3, dtype=bool)
        assert np.max(np.abs((got - UG)[1:-1][..., off])) <= 1e-12 * np.max(np.abs(UG[1:-1][..., off]))
        assert np.max(np.abs((got - UG)[1:-1].imag)) <= 1e-12 * np.max(np.abs(UG[1:-1].imag))


@pytest.mark.parametrize("scale", [1.02, 0.6])
def test_gauge_transformations_off_the_group(oracle, scale):
    """G of equal entries below 1.03, U in SU(3): G U G^dagger has entries up to six."""
    N = (4, 3, 6)
    f = O.random_fields(N, 97, link_amp=0.8, e_amp=0.1)
    G = np.full(O.identity_gauge(N).shape, scale * (1 + 1j))
    H = G.copy()
    st, olog, UG, EG = oracle.coulomb_fix(f, G, N, (1.0, 1.0, 1.0), 1e-3, 1)
    assert st == 0
    with Lattice(N) as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        lat.upload("G", H)
        log = lat.coulomb_fix(1e-3, 1)
        got = {k: lat.download(k) for k in ("G", "UG", "EG")}
    assert np.allclose(log, olog, rtol=1e-11, atol=1e-13)
    for k, want in (("G", G), ("UG", UG), ("EG", EG)):
        assert np.max(np.abs(got[k] - want)[1:-1]) <= 1e-12 * np.max(np.abs(want)), k


@pytest.mark.parametrize("precision,mixed", [("fp64", False), ("fp64", True), ("fp32", False)])
def test_gauge_sweeps_keep_no_memory(precision, mixed):
    """What the sweeps need beyond the handle's fields and transforms is given back (27 doubles a site would be 85 MB here)."""
    torch = pytest.importorskip("torch")
    N = (64, 64, 96)
    with Lattice(N, precision=precision) as lat:
        lat.fill_synthetic(1)
        lat.coulomb_fix(0.08, 0, mixed=mixed)
        lat.synchronize()
        before = torch.cuda.mem_get_info()[0]
        lat.coulomb_fix(0.08, 3, mixed=mixed, open_z=True)
        lat.synchronize()
        assert before - torch.cuda.mem_get_info()[0] < 16 << 20


@pytest.mark.parametrize("N", [(4, 3, 5), (6, 5, 2)])
def test_gauge_sweeps_of_fp32_handles(oracle, N):
    """FP32 handles: the deviations of FP64 arithmetic, links and transformations stored in FP32; the ghost links stay."""
    f = O.random_fields(N, 98, link_amp=0.1, e_amp=0.1)
    with Lattice(N, precision="fp32") as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        held = {k: lat.download(k) for k in ("U", "E")}
        G = O.identity_gauge(N)
        st, olog, UG, EG = oracle.coulomb_fix(held, G, N, (1.0, 1.0, 1.0), 0.08, 2, flags=O.GF_PROJECT_ZERO_MODE)
        log = lat.coulomb_fix(0.08, 2, project_zero_mode=True)
        got = {k: lat.download(k) for k in ("G", "UG", "EG")}
    assert st == 0
    assert np.allclose(log[0], olog[0], rtol=1e-11, atol=1e-13)
    assert np.allclose(log[1], olog[1], rtol=1e-5, atol=1e-6)
    assert np.array_equal(got["UG"][[0, -1]], UG[[0, -1]])
    for k, want in (("G", G), ("UG", UG), ("EG", EG)):
        assert np.max(np.abs(got[k] - want)[1:-1]) <= 5e-7, k


# ---- adjoint: cotangents that are not finite, or of other sizes than the forces they are rotated with
DT = 0.1


def _adjoint(f, N, precision, form):
    with Lattice(N, A, precision=precision) as lat:
        lat.upload_fields(f)
        return lat.adjoint(DT, 2, 3, 6, form, checkpoint_every=1)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_adjoint_keeps_a_nan_to_its_cotangents(precision):
    """A NaN weight on E_x in slices 3 to 5.  The x links of slice 6 get a cotangent only as the far side of the plaquettes
    that begin in slice 5, so two steps' E_x gradient there is NaN through that rotation alone.  Slices the NaN does not
    reach have the gradient of the other weights."""
    N = (4, 5, 12)
    f = O.random_fields(N, 99, link_amp=0.25, e_amp=0.3, j_amp=0.05)
    _, g = _adjoint(f, N, precision, ((float("nan"), 0.5, 0.5, 0.5, 0.5, 0.5), (0,) * 6))
    _, want = _adjoint(f, N, precision, ((0, 0.5, 0.5, 0.5, 0.5, 0.5), (0,) * 6))
    gx = g["E"][1:-1, ..., 0, :]
    assert np.all(np.isnan(gx[3:7]))
    for k in g:
        far = np.r_[1:2, 9:13]
        assert np.all(np.isfinite(g[k][far])), k
        assert np.allclose(g[k][far], want[k][far], rtol=1e-4, atol=1e-6), k


def _gradients_scale(precision, sizes, eps, tiny):
    N = (4, 5, 10)
    f = O.random_fields(N, 100, link_amp=0.25, e_amp=0.3, j_amp=0.05)
    _, want = _adjoint(f, N, precision, ((0.5,) * 6, (0,) * 6))
    for size in sizes:
        _, g = _adjoint(f, N, precision, ((0.5 * size,) * 6, (0,) * 6))
        for k in g:
            top = np.max(np.abs(want[k]))
            assert np.max(np.abs(g[k] / size - want[k])) <= eps * top + 1000 * tiny / size, (k, size)


@pytest.mark.parametrize("precision,sizes", [("fp64", [1e-30, 1e-100, 1e100]), ("fp32", [1e-12, 1e-25, 1e-30, 1e-34, 1e20])])
def test_adjoint_is_linear_in_its_weights(precision, sizes):
    """Cotangents of any size the arithmetic holds give the gradient of weights of one times that size (numbers that
    become subnormal on the way lose what they lose there)."""
    _gradients_scale(precision, sizes, *((1e-12, 5e-324) if precision == "fp64" else (3e-5, 1.4e-45)))


# ---- FP64 numbers below the format's smallest exponents (2^-900, 2^-450 where two exponents add up)
@pytest.mark.parametrize("size", [1e-265, 1e-275, 1e-285, 1e-295])
def test_the_thinnest_slices_keep_their_digits(oracle, size):
    N = (4, 5, 24)
    f = O.random_fields(N, 101, link_amp=0.2, e_amp=0.1, j_amp=0.05)
    far = slice(10, N[2] + 2)
    f["U"][far] = O.new_fields(N)["U"][far]
    f["UOld"] = f["U"].copy()
    for k in ("E", "Jp", "Jm", "JpStat", "JmStat"):
        f[k][far] *= size
    ref = O.copy_fields(f)
    oracle.update(ref, N, A, DT, 2)
    with Lattice(N, A) as lat:
        lat.upload_fields(f)
        lat.step(DT, 2)
        out = lat.download_fields()
        lat.upload("G", _random_gauge(N, 102))
        g = O.links_as_matrices(lat.download("G"))
        lat.coulomb_fix(0.08, 0)
        EG = lat.download("EG")
    want = _rotated(g[..., None, :, :], out["E"])
    for z in range(16, N[2] + 1):  # out of reach of the strong half
        for k in ("E", "Jp", "Jm", "JpStat", "JmStat"):
            assert np.max(np.abs(out[k][z] - ref[k][z])) <= 1e-12 * np.max(np.abs(ref[k][z])), (k, z)
        top = np.max(np.abs(ref["U"][z].imag))
        assert 0 < top < size and np.max(np.abs(out["U"][z].imag - ref["U"][z].imag)) <= 1e-12 * top, z
        assert np.max(np.abs(EG[z] - want[z])) <= 1e-12 * np.max(np.abs(want[z])), z


def test_adjoint_of_the_smallest_weights():
    _gradients_scale("fp64", [1e-130, 1e-145, 1e-160, 1e-250, 1e-290, 1e-306], 1e-12, 5e-324)


# ---- device buffers of the caller, in the middle of an allocation and up to its end
def test_device_buffers_inside_an_allocation():
    torch = pytest.importorskip("torch")
    N = (32, 32, 64)
    f = O.random_fields(N, 103)
    with Lattice(N) as lat:
        n = lat.field_doubles("U")
        block = torch.zeros(n + 1024, dtype=torch.float64, device="cuda")
        lat.synchronize()
        before = torch.cuda.mem_get_info()[0]
        for at in (0, 512, 1024):
            part = block[at:at + n]
            part.copy_(torch.from_numpy(f["U"].view(np.float64).ravel()))
            torch.cuda.synchronize()
            lat.upload_device("U", part.data_ptr())
            lat.synchronize()
            block.zero_()
            torch.cuda.synchronize()
            lat.download_device("U", part.data_ptr())
            assert np.array_equal(part.cpu().numpy(), f["U"].view(np.float64).ravel())
            assert not block[:at].any() and not block[at + n:].any()
        assert before - torch.cuda.mem_get_info()[0] < 8 << 20  # read and written in place: no staging buffer (30 MB)


# ---- gradient arrays: nothing is written to them by the host before the copy that fills or refuses them
DEVICE_GRADIENT = """
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
from oracle import oracle as O
from soerenpragya3dglasma_gb300 import Lattice, _lib
N = (4, 5, 6)
f = O.random_fields(N, 104, link_amp=0.25, e_amp=0.3, j_amp=0.05)
with Lattice(N) as lat:
    lat.upload_fields(f)
    value, want = lat.adjoint(0.1, 2, 1, 5, Lattice.ENERGY, checkpoint_every=1)
    out = torch.zeros(want["E"].size, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    num, den = (ctypes.c_double * 6)(*Lattice.ENERGY[0]), (ctypes.c_double * 6)(*Lattice.ENERGY[1])
    v = ctypes.c_double()
    st = lat.lib.glasma_adjoint(lat.h, 0.1, 2, 1, 1, 5, num, den, ctypes.byref(v),
                                ctypes.cast(out.data_ptr(), _lib._D), None, None, None, None)
    print("status", st)  # refused, or filled
    if st == 0:
        assert np.allclose(out.cpu().numpy(), want["E"].ravel(), rtol=1e-9, atol=1e-12)
    again, _ = lat.adjoint(0.1, 2, 1, 5, Lattice.ENERGY, checkpoint_every=1)
    assert abs(again - value) <= 1e-12 * abs(value)
print("done")
"""


def test_a_device_gradient_array_does_not_end_the_process():
    import os
    import subprocess
    import sys

    pytest.importorskip("torch")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", DEVICE_GRADIENT, root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, (r.returncode, r.stdout, r.stderr[-2000:])


# ---- sums over a slice
def test_a_slice_is_summed_to_its_last_digit():
    """Static currents alone: the violation of a site is -JpStat / sqrt 2 with one rounding, its square's mean over 64 x 64
    sites known in more digits.  One rounding of the result is 5e-17 of it rms (uniform within half a unit, 1.1e-16 at most);
    the sums of a block (128 sites pairwise, 32 blocks averaged) add 1e-17.  32 parts added one after the other would add
    1.5e-16."""
    N = (64, 64, 128)
    f = {"JpStat": O.zero_current(N)}
    f["JpStat"][...] = np.random.default_rng(105).standard_normal(f["JpStat"].shape)
    O.sync_ghosts(f["JpStat"])
    with Lattice(N) as lat:
        lat.upload_fields(f)
        profile = lat.gauss(profile=True)[2]
    G = (f["JpStat"][1:-1] * 0.70710678118654752440).astype(np.longdouble)
    want = np.sum(G * G, axis=(1, 2, 3)) / (N[0] * N[1])
    err = ((profile - want) / want).astype(np.float64)
    assert np.sqrt(np.mean(err ** 2)) < 9e-17


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_a_slice_with_infinities_stays_one(bad):
    N = (4, 3, 5)
    J = O.zero_current(N)
    J[...] = 0.1
    J[3, 1, 2, 4] = bad
    with Lattice(N) as lat:
        lat.upload("JpStat", J)
        profile = lat.gauss(profile=True)[2]
    assert np.array_equal(np.isfinite(profile), np.arange(N[2]) != 2)
    assert np.isnan(profile[2]) if np.isnan(bad) else profile[2] == np.inf


# ---- adjoint on links that are not unitary: a link's variations stay those of the group, whatever the link
@pytest.mark.parametrize("factor", [1.0, 1 + 1e-12, 1 + 1e-6, 1.01, 0.8])
@pytest.mark.parametrize("key", ["E", "Jp"])
def test_adjoint_of_links_off_the_group(factor, key):
    """A fifth of the links scaled: the gradient along a random direction against fourth-order central differences.
    eps = 1e-3 of fields of order one: truncation eps^4 = 1e-12 and rounding 1e-15 / eps = 1e-12 of the objective, which
    is up to a thousand times the derivative: 1e-8 with a margin of ten."""
    N, steps, eps = (4, 5, 10), 3, 1e-3
    rng = np.random.default_rng(106)
    f = O.random_fields(N, 107, link_amp=0.3, e_amp=0.2, j_amp=0.1)
    f["U"][rng.random(f["U"].shape[:3]) < 0.2] *= factor
    O.sync_ghosts(f["U"])
    d = _synced(rng.standard_normal(f[key].shape))

    def value(x):
        with Lattice(N, A) as lat:
            lat.upload_fields(dict(f, **{key: x}))
            lat.step(DT, steps, save_uold=False)
            return lat.objective(2, 8, Lattice.ENERGY)

    with Lattice(N, A) as lat:
        lat.upload_fields(f)
        _, g = lat.adjoint(DT, steps, 2, 8, Lattice.ENERGY, checkpoint_every=1)
    v = [value(f[key] + s * eps * d) for s in (2, 1, -1, -2)]
    fd = (8 * (v[1] - v[2]) - (v[0] - v[3])) / (12 * eps)
    assert abs(fd - float(np.sum(g[key][1:-1] * d[1:-1]))) <= 1e-8 * abs(fd)


def test_fp32_adjoint_of_links_off_the_group():
    """The same links on an FP32 handle: its gradient against the FP64 one of the numbers it holds.  FP32 rounding on hot fields
    is 5e-6 of the gradient after forty steps; three steps stay below 1e-5."""
    N, steps = (4, 5, 10), 3
    rng = np.random.default_rng(108)
    f = O.random_fields(N, 109, link_amp=0.3, e_amp=0.2, j_amp=0.1)
    f["U"][rng.random(f["U"].shape[:3]) < 0.2] *= 0.9
    O.sync_ghosts(f["U"])
    with Lattice(N, A, precision="fp32") as lat:
        lat.upload_fields(f)
        held = lat.download_fields()
        _, g = lat.adjoint(DT, steps, 2, 8, Lattice.ENERGY, checkpoint_every=1)
    with Lattice(N, A) as lat:
        lat.upload_fields(held)
        _, want = lat.adjoint(DT, steps, 2, 8, Lattice.ENERGY, checkpoint_every=1)
    for k in g:
        assert np.max(np.abs(g[k] - want[k])) <= 1e-5 * np.max(np.abs(want[k])), k


@pytest.mark.parametrize("precision,mixed", [("fp64", False), ("fp64", True), ("fp32", False)])
def test_gauge_fields_where_the_guard_ends_the_sweeps(precision, mixed):
    """A NaN link trips the guard: E is left as EG, and UG, whose memory the sweeps use, holds links again: G U G^dagger of the
    transformation the call ends with (mixed: the FP32 sweeps' copy is dropped, so the links themselves)."""
    N = (4, 5, 6)
    f = O.random_fields(N, 110, link_amp=0.1, e_amp=0.1)
    f["U"][2, 1, 2, 0, 0, 0] = np.nan
    with Lattice(N, precision=precision) as lat:
        lat.upload("U", f["U"])
        lat.upload("E", f["E"])
        held = {k: lat.download(k) for k in ("U", "E")}
        with pytest.raises(GlasmaError):
            lat.coulomb_fix(0.08, 5, mixed=mixed)
        got = {k: lat.download(k) for k in ("G", "UG", "EG")}
    assert np.array_equal(got["EG"][1:-1], held["E"][1:-1])
    assert np.array_equal(got["UG"][[0, -1]], O.identity_links(N)[[0, -1]])
    g, u = O.links_as_matrices(got["G"]), O.links_as_matrices(held["U"])
    forward = [np.roll(g, -1, axis=2), np.roll(g, -1, axis=1), np.roll(g, -1, axis=0)]
    for mu in range(3):
        want = g @ u[..., mu, :, :] @ np.swapaxes(forward[mu].conj(), -1, -2)
        if mixed:
            want = u[..., mu, :, :]
        have = O.links_as_matrices(got["UG"])[..., mu, :, :]
        inside = np.s_[1:-2]  # the top slice's z links look at G's ghost
        ok = np.isfinite(want[inside])
        assert np.array_equal(np.isfinite(have[inside]), ok), mu
        assert np.max(np.abs(have - want)[inside][ok], initial=0) <= (1e-13 if precision == "fp64" else 2e-7), mu
