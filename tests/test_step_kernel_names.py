"""Every kernel an instance can report has its own name, and the benchmark labels each."""
import dmm_b200 as dmm

import bench


def test_names_and_labels():
    names = dmm.Instance.STEP_KERNELS
    assert set(names) == set(range(1, 10)) and len(set(names.values())) == len(names)
    assert {k: v for k, v in names.items() if k <= 6} == dmm.Instance.LAUNCH_FORMS
    assert set(names.values()) == set(bench.KERNELS)
    assert set(bench.LARGE_PROFILES) <= set(names.values())
    for summary in bench.LARGE_PROFILES.values():
        assert bench.profiled_traffic(summary) > 0
