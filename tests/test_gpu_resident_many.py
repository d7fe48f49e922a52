"""The resident step kernel against the step graphs where its block and its form
change: more elastic elements than eight lanes each have threads for, more
nodes or searched entries than the smaller block has warps, one issue of many
launches."""
import pytest

from crushrs_b200 import abi, scenarios as S
from tests.test_gpu_resident import _pair, _same

pytestmark = pytest.mark.gpu


def _two_part(n, size=0.15):
    """Two blocks, mostly elastic, behind honeycomb crush zones."""
    def block(mass, n):
        dims = (4 * n * size, n * size, n * size)
        rho = mass / (dims[0] * dims[1] * dims[2])
        return S.vehicle(mass, dims, S.honeycomb(5e6, rho, 0.3e6, 0.2e6, densification=(0.8, 5e6)), crush_zone_length=0.125 * dims[0],
                         body_modulus=2e7, crush_zone_mass=0.1 * mass, crush_element_size=size)

    return S.Model.build(S.scenario(block(2000.0, n), block(1500.0, n), 12.0, 12.0, element_size=size, max_steps=100000))


# 1000 + 7000 and 1452 + 9438 elements (and a road): eight lanes for each elastic
# one and a lane for each of the others are 57,000 and 76,956 threads, the grid has 75,776
@pytest.mark.parametrize("n", [10, 11])
def test_many_elastic_elements(n):
    model = _two_part(n)
    assert model.n_hexes - 8 * n**3 in range(1, 2000)
    _same([model], [40, 85])


@pytest.mark.parametrize("crashes", [7, 30, 110])  # nodes and entries below and above 1184 warps' worth
def test_many_small_crashes(crashes):
    models = [_pair(0.2, 3 + k % 2, layout=abi.LAYOUT_TBONE if k % 3 == 2 else abi.LAYOUT_HEADON) for k in range(min(crashes, 6))]
    _same([models[k % len(models)] for k in range(crashes)], [27, 120])


def test_one_issue_of_many_launches():
    _same([_pair(0.2, 4)], [1100])
