"""A device wait that gives up is not silent: the next verb on the problem and the verbs that wait for the GPU return
TGH_ERR_TIMEOUT until tgh_device_status has reported it, and the problem then works again."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def refuses(tgh, call):
    with pytest.raises(tgh._abi.TGHError) as e:
        call()
    assert e.value.code == tgh._abi.TGH_ERR_TIMEOUT
    assert "gave up" in str(e.value)


# the TMA kernel, and the tile kernel with two staging buffers and with one
@pytest.mark.parametrize("q,N,roots", [(4, 32, 2), (4, 16, 4), (8, 27, 3)])
def test_verbs_refuse_after_a_wait_gave_up(tgh, q, N, roots):
    case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
    f = tgh.gh_forest(case, N, roots)
    P = tgh.GHProblem(case, f, q, margin_check=False, tuned=False)
    Q = tgh.GHProblem(case, f, q, margin_check=False, tuned=False)
    u = P.initial_state(P.statevector(), 0.0)
    du, ref = torch.zeros_like(u), torch.zeros_like(u)
    P.gh_rhs(ref, u, 0.0)
    dt = 0.25 * f.h0 / 4
    for first in (lambda: P.gh_rhs(du, u, 0.0), lambda: P.step_batched(u.clone(), 0.0, dt, 1)):
        P.set_wait_limit(-1)
        first()
        P.set_wait_limit(1 << 26)
        # a verb that waits for the GPU sees the word of the work before it
        refuses(tgh, lambda: P.max_speed(u, 0.0))
        # and so does every verb after, whatever the limit, until the status is read
        for verb in (lambda: P.gh_rhs(du, u, 0.0), lambda: P.step_batched(u.clone(), 0.0, dt, 1),
                     lambda: P.rk4_step(u.clone(), 0.0, dt), lambda: P.prepare(u, 0.0), lambda: P.error_norm(u, 0.0),
                     lambda: P.gh_constraint(u, 0.0), lambda: P.stage_limit(u, 0.0), lambda: P.copy_work(), lambda: P.time_rhs(u, 0.0, nlaunch=1),
                     lambda: Q.transfer_from(P, u, 0.0, du)):
            refuses(tgh, verb)
        refuses(tgh, P.device_status)
        P.device_status()
        P.gh_rhs(du, u, 0.0)
        P.max_speed(u, 0.0)
        assert torch.equal(du, ref)
    P.set_wait_limit(-1)
    refuses(tgh, lambda: P.time_rhs(u, 0.0, nlaunch=1))
    refuses(tgh, P.device_status)
    P.close()
    Q.close()


def test_a_problem_starts_with_a_clean_status(tgh):
    """The status words are lent to one problem after another: what one left behind is not the next one's."""
    case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
    f = tgh.gh_forest(case, 32, 1)
    other = tgh.GHProblem(case, f, 4, margin_check=False)
    for _ in range(3):
        P = tgh.GHProblem(case, f, 4, margin_check=False)
        u = P.initial_state(P.statevector(), 0.0)
        P.max_speed(u, 0.0)
        P.set_wait_limit(-1)
        P.gh_rhs(torch.zeros_like(u), u, 0.0)
        refuses(tgh, lambda: P.max_speed(u, 0.0))
        other.max_speed(u, 0.0)
        P.close()
    other.close()
