"""The one-launch per-atom kernels with networks whose weights are staged in shared
memory (up to 8,192) and read from L2 beyond, against the graph of the batch
kernels, as the other per-atom shapes are."""
import pytest

from tests.test_gpu_atom_edges import test_per_atom_kernels_against_graph as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,arch", [(["Cu"], [40, 56, 51]), (["Cu", "Au"], [62, 57, 3]),
                                        (["Cu"], [64, 64, 64])])
def test_weights_staged_and_not(types, arch, tmp_path):
    check(types, 10, 4, arch, [1] * len(arch) + [0], "current", tmp_path)
