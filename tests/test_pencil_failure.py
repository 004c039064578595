"""What a failed pencil reports: a grid-wide kernel that gave up waiting is not
an overlap that is not positive definite (no GPU needed: the status words are
set here)."""
import ctypes as C

import pytest

import halfb200

GAVE_UP = -100


@pytest.mark.parametrize("infos,words", [
    ((0, 0, 0), ""), ((1, 0, 0), "correction metric"), ((0, 0, 2), "not positive definite (Cholesky info 2)"),
    ((0, 1, 0), "eigensolve failed (info 1)"), ((0, 0, GAVE_UP), "gave up waiting"), ((0, GAVE_UP, 0), "gave up waiting"),
    ((0, GAVE_UP, 1), "gave up waiting")])
def test_failure_text(infos, words):
    lib = C.CDLL(halfb200.library_path())
    text = C.create_string_buffer(256)
    lib.hb_diag_pencil_failure((C.c_int * 3)(*infos), text, 256)
    got = text.value.decode()
    assert words in got if words else got == ""
    assert "positive definite" not in got or GAVE_UP not in infos
