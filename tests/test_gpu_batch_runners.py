"""Batch runners side by side: what one sets up for its molecules, another keeps.

The clustered Lanczos bounds need 24 bytes of shared memory per orbital, more than the default limit
from 2,038 orbitals up. An engine that has taken 2,400 orbitals takes them again after a batch of
2,100 has run beside it.
"""
import pytest

from pm7b200 import api
from pm7b200 import geometry as G

pytestmark = pytest.mark.gpu


def test_a_smaller_batch_does_not_take_the_shared_memory_of_a_larger_one():
    large, small = G.water_cluster(400, seed=1), G.water_cluster(350, seed=2)
    with api.Engine() as eng:
        first = eng.poll(eng.submit(*large, want_matrices=0), wait=True)[1]
        other = api.run_batch([small], want_matrices=0)[0]
        again = eng.poll(eng.submit(*large, want_matrices=0), wait=True)[1]
    for r in (first, other, again):
        assert not isinstance(r, Exception), r
    assert again["total_ev"] == first["total_ev"]
