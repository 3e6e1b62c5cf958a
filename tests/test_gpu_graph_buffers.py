"""Graphs kept by one context over calls whose buffers grow in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_step_calls_of_changing_length():
    """The counts of --two-step grow with the SNPs while the other buffers of the
    graph depend on traits and blocks alone: short, long and short calls again
    return what a context of their own returns."""
    from ldsc_b200.api import Context, h2_batch
    from ldsc_b200.synth import gwas_traits
    rng = np.random.default_rng(3)
    data = {}
    for n in (9_000, 60_000):
        ld = 1.0 + rng.gamma(2.0, 20.0, n)
        data[n] = (*gwas_traits(ld, 2e5, 3, seed=n)[:2], ld, 1.0 + 0.5 * ld)

    def call(c, n, two_step=30.0):
        chi2, ns, ld, wld = data[n]
        return h2_batch(c, chi2, ns, ld, wld, 2e5, 100, two_step=two_step)

    want = {}
    for n in data:
        own = Context(0)
        want[n] = call(own, n)
        own.close()
    c = Context(0)
    call(c, 60_000, None)   # the inputs' buffers at their longest
    for n in (9_000, 60_000, 9_000, 60_000, 9_000):
        got = call(c, n)
        for f in got.dtype.names:
            np.testing.assert_array_equal(got[f], want[n][f])
    c.close()
