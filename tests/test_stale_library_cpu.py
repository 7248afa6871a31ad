"""A kernel library built from other sources than the ctypes binding is refused at load."""
import ctypes as C

import pytest

from fbamtrain_b200.ops import native as nv


def _layout():
    p = nv.GemmParams
    return [C.sizeof(p), p.status.offset, p.out_fp32.offset, p.rs_out.offset, p.rs_row_stores.offset, p.mode.offset,
            p.conv.offset, C.sizeof(nv.ConvGeom)]


class _Library:
    def __init__(self, layout, revision=None):
        def fill(out):
            for i, v in enumerate(layout):
                out[i] = v
        self.fbam_gemm_params_layout = fill
        if revision is not None:
            self.fbam_interface_revision = lambda: revision


def test_matching_library_is_accepted():
    nv._check_struct_layout(_Library(_layout(), nv.INTERFACE_REVISION), "lib")


@pytest.mark.parametrize("revision", [None, 1, 3])
def test_other_revision_is_refused(revision):
    """None: a library from before revisions, whose struct has the same size and the same probed offsets although a field
    was added since (it took the place of padding)."""
    with pytest.raises(RuntimeError, match="different sources"):
        nv._check_struct_layout(_Library(_layout(), revision), "lib")


@pytest.mark.parametrize("i", range(8))
def test_other_layout_is_refused(i):
    layout = _layout()
    layout[i] += 4
    with pytest.raises(RuntimeError, match="different sources"):
        nv._check_struct_layout(_Library(layout, nv.INTERFACE_REVISION), "lib")


def test_built_library_matches():
    if not nv.available():
        pytest.skip("kernel library not built")
    nv.lib()
