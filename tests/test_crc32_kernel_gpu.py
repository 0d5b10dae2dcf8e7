"""The CRC32 kernel at the sizes and addresses where its work is cut: whole 16-byte groups and what is left over at either
end, one CTA against several, one step per thread against many."""
import ctypes
import os
import zlib

import pytest
import torch

pytestmark = pytest.mark.gpu

ONE_CTA = 8 * 256 * 16  # bytes that one CTA still does alone


@pytest.mark.parametrize("offset", [0, 1, 4, 15])
@pytest.mark.parametrize("nbytes", [1, 15, 16, 17, 33, 4095, 4096, 4112, ONE_CTA - 1, ONE_CTA, ONE_CTA + 16, 16 * ONE_CTA + 5, 592 * 256 * 16 * 4 + 16,
                                    64 << 20])
def test_crc32_at_the_cuts(nbytes, offset):
    lib = ctypes.CDLL(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nangila", "libnangila_kernels.so"))
    lib.nangila_crc32_noalloc.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p]
    gen = torch.Generator(device="cuda").manual_seed(nbytes + offset)
    data = torch.randint(0, 256, (nbytes + offset,), dtype=torch.uint8, device="cuda", generator=gen)[offset:]
    out = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    for _ in range(2):  # what the first call left in the result word does not matter to the second
        assert lib.nangila_crc32_noalloc(data.data_ptr(), nbytes, out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        got = out.tolist()
        assert got[0] & 0xFFFFFFFF == zlib.crc32(data.cpu().numpy().tobytes())
        assert got[1] == -1
