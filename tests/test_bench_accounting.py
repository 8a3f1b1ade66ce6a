"""The benchmark's arithmetic on kernel times: no GPU needed."""

import inspect

import bench


def test_rounds_of_a_call_add_up():
    # 20 steps of one compression and two rounds of expansion and attention, of which 30 attention launches were recorded
    ms = bench.kernel_ms_per_step([2.0, 0.0, 8.0, 45.0, 0.0], [20, 0, 40, 30, 0], [1, 0, 2, 2, 0])
    assert ms == [0.1, 0.0, 0.4, 3.0, 0.0]


def test_decode_section_names_its_kernels():
    source = inspect.getsource(bench.decode_section)
    assert '"prepare_queries"' in source and "expand" not in source
