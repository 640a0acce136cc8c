"""The analysis whose weight rows are too many to stage: one and four lanes per output, against the oracle.

T127 with 20 levels has outputs for a lane each and two tables of 103 KB (FP64: 202 KB); with 4 levels four
lanes share an output.  Tolerances: the transforms' own (tests/test_gpu_transforms.py).
"""
import pytest

from jgcm import configs
from test_gpu_transforms import TOL, _grid, _meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nd", [4, 20])
def test_unstaged_analysis(jg, orc, nd, prec):
    gm, om = _meshes(jg, orc, 127, 192, 512, nd, prec)
    u, v = _grid(om, nd, 5), _grid(om, nd, 6)
    for name, ins, n in (("Vor_Div_From_Grid_UV", (u, v), 2), ("Trans_Grid_To_Spherical", (u,), 1)):
        a, b = [gm.spectral(nd) for _ in range(n)], [om.spectral(nd) for _ in range(n)]
        getattr(jg, name)(gm, *ins, *a)
        getattr(orc, name)(om, *ins, *b)
        for x, y in zip(a, b):
            assert configs.rel_l2(x, y) < TOL[prec], name
