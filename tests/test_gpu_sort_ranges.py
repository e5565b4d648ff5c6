"""The pair sort at the edges of its tiles and on both sides of the line
between the small and the large ones: keys and the permutation are a stable
sort's, bit for bit, with keys of one, two and three digits, few distinct
keys, and an explicit payload."""
import ctypes as C

import pytest

import flip2_b200 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 1535, 1536, 1537, 1536 * 9 + 1, 262143, 262144, 262145, 6144 * 60 + 1])
@pytest.mark.parametrize("bits,distinct", [(7, 3), (13, 8192), (20, 1 << 20)])
def test_sort_sizes(n, bits, distinct):
    import torch
    L = F.lib()
    g = torch.Generator(device="cuda").manual_seed(n + bits)
    keys = torch.randint(0, distinct, (n,), device="cuda", dtype=torch.int32, generator=g)
    vals = torch.randint(0, 1 << 30, (n,), device="cuda", dtype=torch.int32, generator=g)
    L.flip_sort_pairs_scratch_bytes.restype = C.c_size_t
    nbytes = L.flip_sort_pairs_scratch_bytes(C.c_uint64(n))
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    want, perm = torch.sort(keys.long(), stable=True)

    def p(t):
        return C.c_void_p(t.data_ptr() if t is not None else None)

    # a scratch sized for more keys holds fewer, and the look-back words of
    # large tiles (1 KB a digit pass and 6144 keys) are enough for any count
    assert L.flip_sort_pairs_scratch_bytes(C.c_uint64(n + 5000)) >= nbytes
    large = nbytes - 4 * 1024 * max(0, -(-min(n, 1 << 18) // 1536) - -(-n // 6144))
    for payload, room in ((None, nbytes), (vals, nbytes), (vals, large)):
        ko, vo = torch.empty_like(keys), torch.empty_like(keys)
        rc = L.flip_sort_pairs(p(keys), p(payload), p(ko), p(vo), C.c_uint64(n), bits, p(scratch), C.c_size_t(room), None)
        torch.cuda.synchronize()
        assert rc == 0
        assert torch.equal(ko.long(), want)
        assert torch.equal(vo.long(), perm if payload is None else vals.long()[perm])
    assert L.flip_sort_pairs(p(keys), None, p(ko), p(vo), C.c_uint64(n), bits, p(scratch), C.c_size_t(large - 1), None) != 0
