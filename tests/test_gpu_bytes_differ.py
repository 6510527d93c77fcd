"""matpl_bytes_differ at the edges of its 16-, 4- and 1-byte paths: lengths around them and around a block's
threads, unaligned starts, a difference in the first, last and a middle byte, answers in pinned and
device memory."""
import pytest
import torch

from matpl_gb300 import _lib
from matpl_gb300._lib import check, ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("off", [0, 4, 1])
@pytest.mark.parametrize("n", [0, 1, 3, 4, 15, 16, 17, 4095, 4096, 16384 + 5, 70001])
def test_differences_are_found(off, n):
    lib, s = _lib.load(), torch.cuda.current_stream().cuda_stream
    a = torch.randint(0, 256, (n + off + 32,), dtype=torch.uint8, device=DEV)
    b = a.clone()
    answers = [torch.full((1,), 7, dtype=torch.int32).pin_memory(), torch.full((1,), 7, dtype=torch.int32, device=DEV)]

    def ask():
        for w in answers:
            check(lib.matpl_bytes_differ(ptr(a) + off, ptr(b) + off, n, ptr(w), s), "matpl_bytes_differ")
        torch.cuda.synchronize()
        return [int(w[0]) for w in answers]
    assert ask() == [0, 0]
    a[off + n:] += 1                             # past the end
    a[:off] += 1                                 # before the start
    assert ask() == [0, 0]
    for q in {0, n // 2, n - 1} if n else ():
        b[off + q] ^= 1
        assert ask() == [1, 1], q
        b[off + q] ^= 1
    assert ask() == [0, 0]
