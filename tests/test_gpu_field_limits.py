"""Fields at the ends of their arguments' ranges: a negative delta (the entry points take any finite
one) beside clusters of no extent."""
import numpy as np
import pytest

from test_gpu_field_far import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nterms", [3, 9, 10])
@pytest.mark.parametrize("scale", [1.0, 1e10])
def test_negative_delta_beside_clusters_of_one_particle(ctx, orc, nterms, scale):
    """A lattice at spacing `scale`, delta = -0.3 scale^2, a particle a leaf: a cluster of no extent
    and a large negative delta.  r^2 of a pair is at least 0.64 scale^2, so r^2 + delta loses
    0.94 / 0.34 = 2.8 of its roundings, and its power 3/2 four: 1e-5 in place of 2e-6."""
    rng = np.random.default_rng(nterms)
    g = np.stack(np.meshgrid(*[np.arange(9.0)] * 3, indexing="ij")).reshape(3, -1)
    x, y, z = (g + rng.uniform(-0.1, 0.1, g.shape)) * scale
    compare(ctx, orc, x, y, z, rng.uniform(-1, 1, g.shape[1]), 1, nterms, 0.5, -0.3 * scale ** 2, 1e-5)
