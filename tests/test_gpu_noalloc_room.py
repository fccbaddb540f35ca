"""wds_forward_noalloc near the end of its fixed array: small networks, whose
top-block inverse takes no room there, and a large one, which keeps only the
pieces of its state there that shared memory does not hold."""
import pytest

from tests.test_zz_no_alloc import _check_calls
from wdsgpu_b200 import GGASolver, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nj,links,B", [(31, 37, 5260), (80, 96, 2908), (3000, 3600, 93)])
def test_batches_the_array_holds(cuda, nj, links, B):
    net = synth.looped_network(3, nj, 1, links)
    s = GGASolver(net, device=cuda, dense_status_machine=True)
    _check_calls(s, net, cuda, [(B, 5), (B // 2, 6)])
