"""gc_gmm_fit at the limits of its inputs."""
import numpy as np
import pytest

from GMM import GMM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 10241])
def test_fit_of_one_colour_with_tiny_covariances(cuda, n, full):
    """Every sample is its component's mean, and the first covariances are so small that any other
    colour (black, say) has density 0: the answer is the colour itself, with covariance min_covar
    after the first step.  Lanes past the last sample take no part in it."""
    colour = np.array([200, 100, 50])
    word = int(colour[0] | colour[1] << 8 | colour[2] << 16)
    g = GMM(3, 1, tolerance=0.0, init_covar=1e-310, full_covariance=full)
    g.fit(np.full(n, word, np.uint32))
    assert g.iterations == 3
    np.testing.assert_array_equal(g.weights, [1.0])
    np.testing.assert_allclose(g.means, [colour], rtol=1e-12)
    # the variance is a difference of numbers up to 200^2, each sum rounded: n * 2^-53 * 200^2
    want = 1e-3 * (np.eye(3)[None] if full else np.ones((1, 3)))
    np.testing.assert_allclose(g.covars, want, rtol=0, atol=n * 2.0 ** -53 * 40000 + 1e-9)


@pytest.mark.parametrize("n", [2 ** 31 - 10000, 2 ** 31 - 4096])
def test_fit_of_nearly_two_to_the_31_samples(cuda, n):
    """Sample counts whose index, a round of the cluster further, does not fit 31 bits (an argument
    holds up to 2^31 - 1): two colours, half the samples each, and one component."""
    torch = cuda
    if torch.cuda.mem_get_info()[0] < 12 << 30:
        pytest.skip("needs 9 GB of free device memory")
    d = torch.full((n,), 10 | 20 << 8 | 30 << 16, dtype=torch.int32, device="cuda")
    d[n // 2:] = 110 | 120 << 8 | 130 << 16
    g = GMM(1, 1, tolerance=0.0)
    g.fit(d)
    assert g.iterations == 1 and g.weights[0] == 1.0
    # sums of n integers are exact below 2^53 / 130^2 terms; the mean of the halves
    np.testing.assert_allclose(g.means, [[60, 70, 80]], rtol=1e-9)
    np.testing.assert_allclose(g.covars, [[2500.001] * 3], rtol=1e-6)
    del d
    torch.cuda.empty_cache()
