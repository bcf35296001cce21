"""The volume kernels a mesh's size chooses between -- the small-mesh kernel
with the face terms, the same after the face kernel, and the kernel with one
thread per tensor line -- against the CPU oracle at sizes on both sides of the
rule, over the branches of the two-point fluxes.  Bar: relative L2 <= 1e-12
per conserved variable (FP64), as for every right-hand side."""
import os
import subprocess

import numpy as np
import pytest

import oracle as O
import theseus_b200 as T
from theseus_b200 import cases
from _helpers import box, oracle_mesh, random_geometry, rel_l2, smooth_state, to_dev

pytestmark = pytest.mark.gpu

TOL = 1e-12
# meshes that take the small-mesh kernel with the face terms, without, and the line kernel
SIZES = {(2, 2): ((9, 7), (97, 95), (147, 149)), (2, 3): ((9, 7), (65, 63), (97, 95)),
         (2, 4): ((9, 7), (41, 39), (73, 71)), (2, 5): ((9, 7), (31, 29), (61, 59)),
         (3, 2): ((3, 4, 5), (14, 15, 13), (19, 17, 18)), (3, 3): ((3, 4, 5), (8, 9, 7), (13, 12, 13)),
         (3, 4): ((3, 4, 5), (8, 7, 9), (10, 9, 11)), (3, 5): ((3, 4, 5), (7, 7, 8), (9, 10, 11))}


def rough_state(m, seed, ratio):
    """Density and pressure jumping by up to `ratio` from node to node."""
    rng = np.random.default_rng(seed)
    shape = (m.num_elements, m.nd)
    s = np.log(ratio)
    return cases.conserved(np.exp(rng.uniform(0, s, shape)), [rng.uniform(-1, 1, shape) for _ in range(m.dim)],
                           np.exp(rng.uniform(0, s, shape)), 1.4)


def compare(m, u, ns, tol=TOL, **kw):
    import torch
    op = (T.NSOperator if ns else T.EulerOperator)(m, **kw)
    ud = to_dev(u, torch.float64)
    du = op.Mult(ud, torch.empty_like(ud)).cpu().numpy()
    cfg = T.make_config(flow="ns" if ns else "euler", volume_flux=kw["numerical_flux"],
                        surface_flux=kw["surface_flux"], **({"mu": kw["mu"]} if ns else {}))
    ref = O.rhs(oracle_mesh(m), cfg, u, nthreads=O.max_threads())
    assert rel_l2(du, ref).max() <= tol, (m.dim, m.order, m.num_elements, kw, rel_l2(du, ref))
    return op


@pytest.mark.parametrize("dim,order", sorted(SIZES))
@pytest.mark.parametrize("size", [0, 1, 2])
def test_volume_kernel_sizes(cuda, dim, order, size):
    m = box(dim, order, SIZES[dim, order][size])
    for vol, surf, ns in (("chandrashekar", "roe", False), ("ranocha", "hll", True), ("hll", "llf", False)):
        kw = dict(numerical_flux=vol, surface_flux=surf, **({"mu": 0.03} if ns else {}))
        compare(m, smooth_state(m, seed=order), ns, **kw)      # both branches of the mean within a line
        nearly = smooth_state(m, seed=order, amp=0.0) * 1e-3   # every mean by its series
        nearly += cases.perturbed_uniform(m.state_shape(), dim, seed=3, amp=0.0)
        compare(m, nearly, ns, **kw)


@pytest.mark.parametrize("size", [1, 2])
@pytest.mark.parametrize("vol", ["chandrashekar", "ranocha"])
def test_far_means_and_scaled_states(cuda, vol, size):
    """Ratios up to 1e6 between neighbours (the logarithm's reduced range), and
    densities and pressures outside the range that the shared reciprocals
    take (2^-100 .. 2^100), where the separate divisions run."""
    m = box(2, 3, SIZES[2, 3][size])
    compare(m, rough_state(m, 1, 1e6), False, numerical_flux=vol, surface_flux="llf")
    # (rho, m, E) -> (a rho, sqrt(ab) m, b E) keeps a state a state
    for a, b in ((2.0 ** -130, 1.0), (1.0, 2.0 ** 130), (2.0 ** 120, 2.0 ** 120)):
        u = rough_state(m, 2, 3.0)
        u[0] *= a
        u[1:3] *= np.sqrt(a * b)
        u[3] *= b
        compare(m, u, False, numerical_flux=vol, surface_flux="llf")


def test_shared_reciprocals_and_logarithm(cuda, tmp_path):
    """Quotients, logarithmic means and fluxes formed from shared reciprocals
    equal the separately divided ones on 19 million seeded samples (a sample
    differs with probability below 2^-34); the logarithm of the far means is
    within one ulp, CUDA's documented bound for log(), and on average as far
    off as log() (to 1 %: the two round 2^20 samples differently)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe, out = str(tmp_path / "check"), str(tmp_path / "logs")
    subprocess.check_call(
        ["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
         "--fmad=false", "--expt-relaxed-constexpr", "-I", os.path.join(root, "theseus_b200", "csrc"),
         "-I", os.path.join(root, "include"), os.path.join(root, "tests", "cpp", "shared_reciprocals_check.cu"),
         "-o", exe], stderr=subprocess.DEVNULL)
    r = subprocess.run([exe, out], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    x, own, cuda_log = np.fromfile(out).reshape(-1, 3).T
    ref = np.log(x.astype(np.longdouble))
    some = x != 1.0
    ulp = np.ldexp(1.0, np.frexp(ref[some].astype(float))[1] - 53)
    err = lambda v: np.abs((v[some] - ref[some]).astype(float)) / ulp  # noqa: E731
    assert (own[~some] == 0.0).all()
    assert err(own).max() <= 1.0 and err(own).mean() <= 1.01 * err(cuda_log).mean(), \
        (err(own).max(), err(own).mean(), err(cuda_log).max(), err(cuda_log).mean())
    print("log_normal", err(own).max(), err(own).mean(), "log", err(cuda_log).max(), err(cuda_log).mean())


@pytest.mark.parametrize("size", [1, 2])
def test_general_geometry(cuda, size):
    m = random_geometry(box(3, 3, SIZES[3, 3][size]), seed=4)
    compare(m, smooth_state(m, seed=2), True, numerical_flux="ranocha", surface_flux="roe", mu=0.02)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_small_mesh_stages_do_not_read_what_they_write(cuda, precision):
    """The small-mesh kernel reads its neighbours' states while other CTAs
    write theirs: the stages alternate between buffers, so every repetition of
    a run gives the same bits, and those of a composed FP64 step."""
    import torch
    m = box(2, 3, (46, 47))
    op = T.EulerOperator(m, numerical_flux="chandrashekar", surface_flux="roe", precision=precision,
                         state_offset=[1.0, 0, 0, 2.5] if precision == "fp32" else None)
    u0 = to_dev(smooth_state(m, seed=1), torch.float64)
    runs = [op.rk3_steps(u0.clone(), 1e-4, 40) for _ in range(6)]
    assert all(torch.equal(runs[0], r) for r in runs[1:])
    if precision == "fp64":
        u, dt, k = u0.clone(), 1e-4, torch.empty_like(u0)
        for _ in range(3):
            y = u + dt * op.Mult(u, k)
            y = 0.75 * u + 0.25 * (y + dt * op.Mult(y, k))
            u = (1.0 / 3.0) * u + (2.0 / 3.0) * (y + dt * op.Mult(y, k))
        v = op.rk3_steps(u0.clone(), 1e-4, 3)
        assert (u - v).abs().max() <= 8 * np.finfo(float).eps * u.abs().max()


def test_rate_over_its_state(cuda):
    """A rate written over its state, as the separate kernels allow it."""
    import torch
    m = box(2, 3, (40, 40))
    op = T.EulerOperator(m, numerical_flux="ranocha", surface_flux="hll")
    u = to_dev(smooth_state(m, seed=5), torch.float64)
    ref = op.Mult(u, torch.empty_like(u))
    assert torch.equal(op.Mult(u, u), ref)


@pytest.mark.parametrize("order,n", [(2, (4, 3, 4)), (4, (3, 4, 3)), (5, (3, 3, 3))])
def test_viscous_rate_over_its_state(cuda, order, n):
    """The same for Navier-Stokes: a mesh of the fused kernel falls back on the
    gradient, face and volume kernels of the larger meshes, which an operator of
    its size launches only here."""
    import torch
    m = box(3, order, n)
    op = T.NSOperator(m, numerical_flux="ranocha", surface_flux="hll", mu=0.02)
    u = to_dev(smooth_state(m, seed=5), torch.float64)
    ref = op.Mult(u, torch.empty_like(u))
    assert torch.equal(op.Mult(u, u), ref) and op.read_status() == 0


@pytest.mark.parametrize("dim,order", sorted(SIZES))
def test_metric_per_node(cuda, dim, order):
    """Metrics that vary within the element, by the line kernel, on both of its
    paths; one of all elements alike too (an element stride of zero)."""
    m = random_geometry(box(dim, order, SIZES[dim, order][2]), seed=order)
    nearly = cases.perturbed_uniform(m.state_shape(), dim, seed=3, amp=1e-3)
    for vol, surf, ns in (("chandrashekar", "roe", False), ("ranocha", "hll", True), ("hll", "llf", False)):
        kw = dict(numerical_flux=vol, surface_flux=surf, **({"mu": 0.03} if ns else {}))
        compare(m, smooth_state(m, seed=order), ns, **kw)
        compare(m, nearly, ns, **kw)
    m.metric[...] = m.metric[:1]
    compare(m, smooth_state(m, seed=order), True, numerical_flux="ranocha", surface_flux="hll", mu=0.03)


@pytest.mark.parametrize("dim,order", sorted(SIZES))
@pytest.mark.parametrize("size", [0, 1, 2])
def test_fp32_sizes(cuda, dim, order, size):
    """FP32-mixed on the same meshes.  Euler, neighbouring nodes' densities and
    pressures up to 8 % apart: a rate sums differences of fluxes that a few
    roundings of 6e-8 each enter, 3e-7 of the rate at most where every
    logarithmic mean is as good (bar 5e-7; means from the rounded ratio's
    logarithm are off by 1e-6).  Navier-Stokes on boxes along the axes: the bar
    of the FP32 right-hand sides, 2e-5."""
    import torch
    m = box(dim, order, SIZES[dim, order][size])

    def error(u, ns, vol, surf, **kw):
        off = [float(u[k].mean()) for k in range(dim + 2)]
        o = np.array(off).reshape(-1, 1, 1)
        u = (u - o).astype(np.float32).astype(np.float64) + o  # what the working copy holds
        op = (T.NSOperator if ns else T.EulerOperator)(m, numerical_flux=vol, surface_flux=surf, precision="fp32",
                                                       state_offset=off, **kw)
        ud = to_dev(u, torch.float64)
        du = op.Mult(ud, torch.empty_like(ud)).cpu().numpy()
        cfg = T.make_config(flow="ns" if ns else "euler", volume_flux=vol, surface_flux=surf, **kw)
        return rel_l2(du, O.rhs(oracle_mesh(m), cfg, u, nthreads=O.max_threads())).max()

    for vol, surf in (("ranocha", "llf"), ("chandrashekar", "roe"), ("hll", "hll")):
        assert error(rough_state(m, order, 1.08), False, vol, surf) <= 5e-7, (vol, surf)
    assert error(smooth_state(m, seed=order), True, "ranocha", "hll", mu=0.01) <= 2e-5
