"""qcs_cuda_sample_noalloc on a caller's own buffer: a slice of a complex64 tensor
lies on 8 bytes, which states below a full sampling tile (4096 amplitudes) take;
what the kernels cannot read is refused before any launch.

Tolerance: none.  The same amplitudes at 16 bytes give the same indices."""
import ctypes as C

import numpy as np
import pytest

from qcs_gb300 import capi


@pytest.mark.parametrize("prec,count,offset", [
    (capi.C64, 4, 4), (capi.C64, 2048, 12), (capi.C64, 4096, 8), (capi.C64, 1 << 20, 8),
    (capi.C128, 1, 8), (capi.C128, 64, 4), (capi.C128, 8192, 8)])
def test_refuses_what_it_cannot_read(prec, count, offset):
    buf = np.zeros(4096, dtype=np.float64)  # host memory: never read
    at = (buf.ctypes.data + 15) // 16 * 16 + offset
    rc = capi.lib().qcs_cuda_sample_noalloc(C.c_void_p(at), count, prec, None, 0, None, None)
    assert rc == capi.EINVAL
    assert b"aligned" in capi.lib().qcs_cuda_last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 2, 4, 8, 64, 128, 256, 1024, 2048])
def test_complex64_states_on_8_bytes(count):
    torch = pytest.importorskip("torch")
    r = np.random.default_rng(count)
    a = (r.normal(size=count) + 1j * r.normal(size=count)).astype(np.complex64)
    a /= np.float32(np.linalg.norm(a))
    draws = torch.from_numpy(r.random(777)).to("cuda")
    got = []
    for skip in (0, 1):
        buf = torch.zeros(count + 2, dtype=torch.complex64, device="cuda")
        v = buf[skip:skip + count]
        v.copy_(torch.from_numpy(a))
        assert v.data_ptr() % 16 == 8 * skip
        out = torch.full((777,), -7, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        rc = capi.lib().qcs_cuda_sample_noalloc(
            C.c_void_p(v.data_ptr()), count, capi.C64, C.c_void_p(draws.data_ptr()), 777,
            C.c_void_p(out.data_ptr()), None)
        assert rc == capi.OK, capi.lib().qcs_cuda_last_error()
        torch.cuda.synchronize()
        got.append(out.cpu().numpy())
    assert np.array_equal(got[0], got[1])
    assert np.all(got[0] < count) and np.mean(got[0] >= 0) > 0.98
