"""What a bounded wait that gave up reports: kernels wait for their own
shared-memory copies, and the CTAs of step_loop for one another."""
import ctypes as C

from fortran_loadfile_mitiwing_b200 import _abi


def test_timeout_message_names_both_waits():
    lib = _abi.load_library()
    buf = C.create_string_buffer(256)
    assert lib.lbm_describe_status(_abi.LBM_ST_TIMEOUT, buf, 256) == _abi.LBM_ERR_CUDA
    text = buf.value.decode()
    assert "shared-memory copy" in text and "step_loop" in text
