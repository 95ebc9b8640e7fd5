"""What the autotuner times and what its results stand for: below 65,000 nucleotides the two pair-block sizes of a
shape launch the same kernels, so only the first is timed and chosen; and a result is not taken over the bound
from which they differ, although both sides have the same power of two of nucleotides."""
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G

pytestmark = pytest.mark.gpu


def _tuned(n, **kw):
    s = G.system_for_config(1, seed=41, scale=n / 40000.0)
    m = MDSystem(s.box, s.top, dna2_settings(s.T, 0.5), md_settings(autotune=True, **kw))
    m.set_state(s.pos, s.quats(), s.vel, s.L)
    shape = m.force_shape()
    m.close()
    return shape


@pytest.mark.parametrize("n", [600, 3000, 13000, 24000])
@pytest.mark.parametrize("precision", ["mixed", "float"])
def test_equal_shapes_are_one(n, precision):
    # sizes of classes of their own (powers of two)
    assert _tuned(n, precision=precision)["pair_npw"] == 32


def test_a_result_stays_below_the_bound():
    below, again, above = _tuned(64000), _tuned(64400), _tuned(65400)
    assert again == below  # taken from the cache: the very same time
    assert above["launch_us"] != below["launch_us"]
