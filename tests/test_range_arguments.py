"""Argument checks of the bitmap factorize that come before any device call: a
range that its workspace query rejects is refused whatever the workspace (no GPU,
no memory touched)."""

import pytest


@pytest.mark.parametrize("span", [0, -1, 2 ** 40, 2 ** 62])
def test_range_is_refused(span):
    from hdfe_stream_b200 import _lib
    lib = _lib.lib()
    assert lib.hdfe_factorize_range_workspace_bytes(span) == -1
    st = lib.hdfe_factorize_range(256, 8, 10, 0, span, 256, 256, 256, 256, 2 ** 62, None)
    assert st == _lib.HDFE_ERR_ARG


def test_small_workspace_is_refused():
    from hdfe_stream_b200 import _lib
    lib = _lib.lib()
    need = lib.hdfe_factorize_range_workspace_bytes(1000)
    st = lib.hdfe_factorize_range(256, 8, 10, 0, 1000, 256, 256, 256, 256, need - 1, None)
    assert st == _lib.HDFE_ERR_WORKSPACE
