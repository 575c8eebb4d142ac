"""bench.py's FP64 roofline of the factored plain step: the work per membrane
depends on the tile size, so only a count of the size that ran is used."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

PEAK = {'warp_inst_per_s': 16.0e9, 'fma_tflops': 1.024, 'ms': 10.0, 'launch': 'probe'}


def test_the_size_that_ran():
    counts = json.load(open(os.path.join(ROOT, 'profiles', 'fp64_counts.json')))['kernels']
    for workload, kernels in counts.items():
        for name, e in kernels.items():
            if name.startswith('k_plain_step'):
                r = bench.fp64_roofline(0.02, 1000, PEAK, name, workload)
                per_mem = e['fp64_warp_inst_per_launch'] / e.get('steps_per_launch', 1) / e['membranes']
                assert 'count_of' not in r
                assert r['achieved'] == pytest.approx(per_mem * 1000 / 0.02e-3 / 1e9), (workload, name)


@pytest.mark.parametrize('kernel', ['k_plain_step (1 cells)', 'k_plain_step (128 cells)'])
def test_another_size_has_no_count(kernel):
    for workload in ('plain250', 'cluster100k', 'no-such-workload'):
        r = bench.fp64_roofline(0.02, 1426, PEAK, kernel, workload)
        assert r['achieved'] is None and r['frac'] is None, workload
