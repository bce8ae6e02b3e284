"""The update percentage of parallel ICD iterations, which is their stop
statistic, against the column kernel's first schedule.

Columns in flight read each other's stale error sinogram, so an iteration's
result depends on how many there are and on how long each of them holds what it
has read.  PCT holds the mean and the run-to-run standard deviation, in
percent, of iterations 2 to 8 over 64 runs with that schedule: CTAs of 64, 128
or 256 threads, as many as are resident and no more than one column in 32, the
short items eight at a time.

Tolerance: the mean over the seven iterations of (shift / spread) stays within
1.5: one spread of a single run, and a margin for the standard errors of the
means of 40 and 64 runs (a run's mean over its iterations varies by 0.5 to 0.6,
so 0.11 together).  Twice as many columns in flight move it by 3 to 9.
"""
import numpy as np
import pytest

import common
import xtg

pytestmark = pytest.mark.gpu

PCT = {
    # N, rows, frames, views: means, standard deviations
    (64, 8, 4, 192): ([18.586, 7.7458, 2.7472, 1.4367, 0.69942, 0.32574, 0.16803],
        [0.02109, 0.008376, 0.003868, 0.002264, 0.001273, 0.0006151, 0.0003331]),
    (80, 8, 1, 200): ([17.148, 4.593, 1.4537, 0.64655, 0.307, 0.12508, 0.073828],
        [0.03442, 0.01096, 0.004046, 0.002343, 0.001175, 0.0004603, 0.0003131]),
    (72, 27, 1, 300): ([16.524, 5.4589, 1.8424, 0.92237, 0.54984, 0.27557, 0.13322],
        [0.02829, 0.009921, 0.004149, 0.00247, 0.001848, 0.0009142, 0.0004959]),
    (96, 16, 4, 384): ([15.482, 4.9403, 1.734, 0.79427, 0.35706, 0.16209, 0.082533],
        [0.01097, 0.004036, 0.001768, 0.001002, 0.0005265, 0.0002817, 0.0001638]),
    (96, 32, 8, 512): ([16.657, 5.9022, 2.403, 1.1527, 0.54053, 0.27657, 0.14644],
        [0.007133, 0.00261, 0.001192, 0.0007385, 0.000378, 0.0002414, 0.0001512]),
    (100, 8, 4, 256): ([15.203, 4.6955, 1.7824, 0.76343, 0.32391, 0.16312, 0.074563],
        [0.01358, 0.005374, 0.002241, 0.001221, 0.002566, 0.0006395, 0.0001978]),
}


def run(case, reps, engine=xtg):
    """[reps][iterations 1..8] update percentages of a reconstruction from a noisy phantom."""
    N, NT, n_time, NP = case
    p = common.params(N=N, NT=NT, NP=NP, n_time=n_time, zinger=True, nhicd=True)
    t, a = common.views(p, (8, NP // n_time // 2) if n_time > 1 else None)
    x0, _, y, w = common.data(p, t, a, seed=4, zfrac=0.005)
    xs = np.maximum(x0 + np.random.default_rng(8).normal(0, 2e-4, x0.shape), 0).astype(np.float32)
    ctx = engine.Context(p, t, a)
    ctx.set_options(a_mode=xtg.XTG_A_TABLE32)
    ctx.upload_sino(y, w)
    out = []
    for _ in range(reps):
        ctx.upload_object(xs)
        ctx.init_error_sino()
        out.append([ctx.iteration(it).avg_update_pct for it in range(1, 9)])
    ctx.close()
    return np.array(out)


@pytest.mark.parametrize("case", sorted(PCT))
def test_update_percentage(case):
    mean, spread = (np.array(v) for v in PCT[case])
    got = run(case, 40)[:, 1:].mean(0)
    assert abs(np.mean((got - mean) / spread)) <= 1.5
