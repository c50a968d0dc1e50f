"""pcs_kernel_stats.kernel_launches: nine kernels a round, ten where the row
kernel with double sums is followed by the launch for what it leaves."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,double,kernels", [(64, 0, 9), (64, 1, 9), (500, 0, 9), (500, 1, 10)])
def test_kernels_per_round(pcs, bins, double, kernels):
    import part_conc_spt_abc_gb300.workloads as W
    with pcs.Context(0) as c:
        inp, _ = W.make_problem(c, [150.0], [10.0], 5e13, [1.0], 3, 40, bins, 24, 1)
        inp.params.avg_trial_count = 50
        inp.params.distance_double = double
        sim = pcs.make_simulation(c, inp, 1)
        c.reset_kernel_stats()
        sim.run()
        k = c.kernel_stats()
        sim.close()
    assert k.rounds > 0 and k.kernel_launches == kernels * k.rounds
