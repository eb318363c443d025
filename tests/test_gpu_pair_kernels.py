"""Every instance of the two pair kernels (a warp per tile, and a thread block per tile for small systems) against the
FP64 oracle: with and without the class-pair table, gates and scales, soft core, switching function and order-2 overlap,
on both sides of the size where the kernel changes (6,144 particles)."""
import numpy as np
import pytest

from interaxplugin import workloads as W
from parity import compare

pytestmark = pytest.mark.gpu

OPTIONS = {
    "uniform table": dict(),
    "scaled table": dict(alchemical_waters=range(0, 40, 3)),
    "uniform parameters": dict(distinct=20),
    "scaled parameters": dict(distinct=20, alchemical_waters=range(0, 40, 3)),
    "soft core and switch, table": dict(alchemical_waters=range(0, 40, 3), softcore_radius=0.1, use_switch=True,
                                        switch_distance=0.7),
    "soft core, switch, order-2 overlap": dict(distinct=20, alchemical_waters=range(0, 40, 3), softcore_radius=0.1,
                                               use_switch=True, switch_distance=0.7, overlap_method=2),
}


@pytest.mark.parametrize("options", OPTIONS)
@pytest.mark.parametrize("waters", [216, 2048, 2049])
def test_instance_against_the_oracle(waters, options):
    kw = OPTIONS[options]
    system, pos, box = W.water_box(waters, W.box_length_for(waters), 0.85, seed=waters, three_body=False, **kw)
    parameters = {"lambda_sterics": 0.6} if "alchemical_waters" in kw else None
    # on the reference's error scale (the sum of |pair energies|): the terms of a random box can cancel in the total
    compare(system, pos, box, parameters, scale="abs")
