"""The convolution entry points refuse tensors that do not start on 16 bytes
before they launch anything (their kernels move 16 bytes at a time; a misaligned
load would fault on the device).  Checked without a device: a refused call never
looks at its pointers."""

import ctypes

import pytest

OK = 1 << 20


@pytest.mark.parametrize("bad", range(3))
def test_misaligned_tensors_are_refused(lib, bad):
    from voxelsim_fea_b200 import _lib
    p = [ctypes.c_void_p(OK + (2 if k == bad else 0)) for k in range(3)]
    work = ctypes.c_void_p(OK)
    assert lib.vf_nn_conv3d_forward(p[0], p[1], None, None, 0, p[2], None, 4, 4, 4, 16, 16, None) == _lib.VF_ERR_ARG
    assert lib.vf_nn_conv3d_forward(p[0], p[1], None, None, 0, None, p[2], 4, 4, 4, 16, 16, None) == _lib.VF_ERR_ARG
    assert lib.vf_nn_conv3d_backward_data(p[0], p[1], None, p[2], 4, 4, 4, 16, 16, None) == _lib.VF_ERR_ARG
    if bad < 2:
        assert lib.vf_nn_conv3d_backward_weight(p[0], p[1], work, 0, work, 1 << 20, 4, 4, 4, 16, 16,
                                                None) == _lib.VF_ERR_ARG
    if bad == 0:
        assert lib.vf_nn_conv3d_backward_bias(p[0], work, work, 1 << 20, 64, 16, None) == _lib.VF_ERR_ARG
