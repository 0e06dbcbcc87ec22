"""The FP64 server and its lattices' fixed-point links under the HBM budget.

Tolerance: solutions meet their 1e-10, so two of them differ by at most
100 * tol as in the server's other tests."""
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
DIMS = (8, 4, 4, 8)


# requests that fit the budget beside the fixed-point links: one and a half (the
# second waits and the links stay, though both requests fit without them), or
# half of one (the links go for the first)
@pytest.mark.parametrize("beside, kept", [(1.5, True), (0.5, False)])
def test_waiting_requests_do_not_cost_the_links(wd, ctx, beside, kept):
    gauge = wd.gen_gauge(DIMS, seed=41)

    def serve(budget, check):
        sv = wd.Server(ctx, prec=wd.F64, hbm_budget_bytes=budget)
        lat = sv.add_lattice(DIMS, gauge)
        _, _, links = sv.status()
        rids = [sv.submit(lat, 1, mass=0.1, tol=1e-10, seeds=[k]) for k in (5, 6)]
        sv.step()
        check(sv, links)
        out = {}
        for _ in range(20):
            for r in rids:
                if r not in out:
                    done, sols, stats, _ = sv.poll(r, want_solutions=True)
                    if done:
                        assert stats[0].converged and stats[0].true_residual <= 1e-10
                        out[r] = sols[0]
            if len(out) == 2:
                break
            sv.step()
        sv.close()
        return [out[r] for r in rids], links

    seen = {}
    free, links = serve(150e9, lambda sv, n: seen.update(used=sv.status()[2]))
    request = (seen["used"] - links) / 2  # both are admitted at once
    fix = DIMS[0] * DIMS[1] * DIMS[2] * DIMS[3] * 4 * 9 * 16

    def check(sv, _):
        queued, _, used = sv.status()
        assert queued == 1
        assert used == links + request - (0 if kept else fix)

    tight, _ = serve(links + beside * request, check)
    for a, b in zip(free, tight):
        assert rel_l2(a, b) <= 100 * 1e-10
