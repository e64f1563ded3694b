"""The tile kernels' shared memory, checked on the host for every kind of the
tile kernels: compiles tests/tile_kinds_check.cu (host code only) with the
library's own flags and runs it."""

from __future__ import annotations

from test_tile_numbers import run_host_check


def test_shared_memory_of_every_tile_kind(tmp_path):
    run_host_check("tile_kinds_check", tmp_path)
