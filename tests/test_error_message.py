"""The message of a failed call stays until the caller reads it, whatever handles
a garbage collector releases in between."""
from __future__ import annotations

import ctypes as C

import pytest


@pytest.mark.parametrize("release", ["pc_graph_destroy", "pc_pgraph_destroy", "pc_batch_destroy", "pc_host_csr_free"])
def test_release_keeps_the_message(pc, release):
    from partitionandconquer_b200 import _lib
    out = C.c_void_p()
    assert _lib.lib.pc_graph_create(None, None, None, 3, 0, 0, C.byref(out)) != 0
    assert b"csr_vlist" in _lib.lib.pc_last_error()
    assert getattr(_lib.lib, release)(None) == 0
    assert b"csr_vlist" in _lib.lib.pc_last_error()
