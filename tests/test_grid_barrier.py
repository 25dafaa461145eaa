"""The grid barrier of the cooperative kernels, replayed on the CPU in random order:
every CTA finds a flag exactly where one was raised."""
from test_index_math import _run


def test_flags_are_found_where_they_were_raised(tmp_path):
    _run('barrier_check', tmp_path)
