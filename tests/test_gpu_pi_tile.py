"""The tile Pi kernel against the one-point kernel, bit for bit, where its tiles can go wrong: rows, planes and the
second point of a pair past a block's end (odd and even edges, 9 to 96), the smallest and largest halos (q = 2 and
8), one staging buffer and two, blocks that keep all, some or none of their upper faces, a layer and a frozen core,
no dissipation. The meshes hold enough points for the kernel to be the one that runs, which every case checks."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

# q, N, roots; periodic gauge wave
WAVES = [(2, 31, 3), (2, 32, 3), (4, 9, 6), (4, 10, 5), (4, 16, 3), (4, 27, 2), (4, 33, 2), (6, 13, 4), (6, 24, 2),
         (8, 12, 4), (8, 21, 3), (8, 96, 1)]


def _both(tgh, case, forest, q, steps=True):
    P = tgh.GHProblem(case, forest, q, margin_check=False, tuned=False)
    assert P.variant()["pi"] == "tile"
    assert P.pi_kernel("plain") == "tile" and P.pi_kernel("plain", "l1") == "l1"
    if steps:
        assert P.pi_kernel("batched") == "tile" and P.pi_kernel("batched", "l1") == "l1"
    g = torch.Generator(device="cuda").manual_seed(11)
    u = P.initial_state(P.statevector(), 0.0)
    u += 1e-6 * torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=g)
    outs = []
    for pi in ("l1", "tile"):
        P.set_variant(pi=pi)
        du = torch.full_like(u, float("nan"))
        P.gh_rhs(du, u, 0.0)
        a = u.clone()
        if steps:
            P.step_batched(a, 0.0, 1e-4, 2)
        P.device_status()
        outs.append((du, a))
    assert torch.isfinite(outs[0][0]).all() and torch.isfinite(outs[0][1]).all()
    assert torch.equal(outs[0][0], outs[1][0])
    assert torch.equal(outs[0][1], outs[1][1])
    P.close()


@pytest.mark.parametrize("q,N,roots", WAVES)
@pytest.mark.parametrize("eps", [0.5, 0.0])
def test_tile_kernel_gives_the_one_point_kernels_bits(tgh, q, N, roots, eps):
    case = tgh.gauge_wave_case(eps_ko=eps, gamma0=1.0)
    _both(tgh, case, tgh.gh_forest(case, N, roots), q)


@pytest.mark.parametrize("q", [2, 4, 6])
def test_tile_kernel_on_blocks_of_8_in_the_plain_form(tgh, q):
    case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
    _both(tgh, case, tgh.gh_forest(case, 8, 9 if q == 2 else 4), q, steps=False)


def test_the_rules_line(tgh):
    """Which kernel a mesh runs on either side of the line, in both forms, and at N = 32, q = 4."""
    case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
    for q, N, roots, plain, batched in ((4, 12, 2, "l1", "l1"), (4, 16, 2, "tile", "l1"), (4, 16, 3, "tile", "tile"),
                                        (4, 8, 5, "tile", "l1"), (2, 16, 4, "l1", "l1"), (2, 32, 3, "tile", "tile"),
                                        (4, 32, 1, "tma", "tma")):
        P = tgh.GHProblem(case, tgh.gh_forest(case, N, roots), q, margin_check=False, tuned=False)
        assert (P.pi_kernel("plain"), P.pi_kernel("batched")) == (plain, batched), (q, N, roots)
        assert P.computed_points() == ((N + 1) ** 3 if roots == 1 else (N * roots) ** 3)
        P.close()


@pytest.mark.parametrize("variant", ["damped", "frozen", "pasted"])
@pytest.mark.parametrize("q,N", [(4, 16), (6, 15)])
def test_tile_kernel_around_an_interior(tgh, variant, q, N):
    case = tgh.kerr_schild_case(a=0.7, halfwidth=3.0, variant=variant)
    _both(tgh, case, tgh.gh_forest(case, N, 4), q, steps=variant != "pasted")


def test_tile_kernel_on_refined_blocks(tgh):
    case = tgh.kerr_schild_case(a=0.7, v=0.1, halfwidth=4.0, gauge="algebraic")
    _both(tgh, case, tgh.hole_forest(case, 16, 4, [2.0]), 4)


def test_tile_variant_is_refused_where_it_does_not_apply(tgh):
    for q, N, precision in ((4, 32, "fp64"), (4, 16, "mixed"), (2, 98, "fp64")):
        case = tgh.gauge_wave_case(eps_ko=0.5)
        P = tgh.GHProblem(case, tgh.gh_forest(case, N, 1), q, margin_check=False, precision=precision, tuned=False)
        with pytest.raises(tgh._abi.TGHError) as e:
            P.set_variant(pi="tile")
        assert e.value.code == tgh._abi.TGH_ERR_ARG
        P.close()


@pytest.mark.parametrize("limit", [-1, -2])
@pytest.mark.parametrize("q,N", [(4, 16), (8, 27)])
def test_a_tile_wait_that_runs_out_is_reported(tgh, q, N, limit):
    """With two staging buffers (q = 4) and with one (q = 8): every CTA gives up on the first of its first two copies,
    or (limit -2) on the second, when h's box may have been refilled already; it lets the copies that it issued land
    and leaves at once: a wait for a copy never issued would go on for 2^24 polls."""
    case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
    P = tgh.GHProblem(case, tgh.gh_forest(case, N, 3), q, margin_check=False, tuned=False)
    u = P.initial_state(P.statevector(), 0.25)
    ref, du = torch.zeros_like(u), torch.zeros_like(u)
    P.gh_rhs(ref, u, 0.25)
    P.set_wait_limit(limit)
    took = []
    for _ in range(3):
        torch.cuda.synchronize()
        start = time.perf_counter()
        P.gh_rhs(du, u, 0.25)
        with pytest.raises(tgh._abi.TGHError) as e:
            P.device_status()
        took.append(time.perf_counter() - start)
        assert e.value.code == tgh._abi.TGH_ERR_TIMEOUT
    # the launches take under a millisecond, 2^24 polls 0.4 s at the least (50 cycles each at 1.965 GHz); the quickest of
    # three, as the host may be held up in one
    assert min(took) < 0.2
    P.set_wait_limit(1 << 26)
    P.gh_rhs(du, u, 0.25)
    P.device_status()
    assert torch.equal(du, ref)
    P.close()
