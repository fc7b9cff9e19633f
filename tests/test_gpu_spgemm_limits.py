"""GPU limits of the sparse product: the longest row that is counted in 32 bits, and
columns that a matrix without columns cannot have."""
import pytest

pytestmark = pytest.mark.gpu
NOT_SUPPORTED, INVALID_INDEX = 8, 9


# one row of A names one row of B many times over: 2^32 - 1024 candidates (one more than the
# kernels take) and 2^32 - 4; the row is refused before any kernel walks it
@pytest.mark.parametrize("dtype", ["float32", "int32"])
@pytest.mark.parametrize("entries,length", [(1024, (1 << 22) - 1), (1023, (1 << 32) // 1023)])
def test_row_past_32_bits_is_refused(b2, cuda, dtype, entries, length):
    torch = cuda
    assert (1 << 32) - 1024 <= entries * length < 1 << 32
    dt = getattr(torch, dtype)
    arp = torch.tensor([0, entries], dtype=torch.int64, device="cuda")
    aci = torch.zeros(entries, dtype=torch.int32, device="cuda")
    brp = torch.tensor([0, length], dtype=torch.int64, device="cuda")
    bci = torch.arange(length, dtype=torch.int32, device="cuda").remainder_(1000)
    with pytest.raises(b2.B2Error) as e:
        b2.minplus_spgemm((arp, aci, torch.ones(entries, dtype=dt, device="cuda"), 1),
                          (brp, bci, torch.ones(length, dtype=dt, device="cuda"), 1000))
    assert e.value.status == NOT_SUPPORTED


# B has entries but no columns: every one of them is out of range, also where A's rows are
# all long (more than 512 candidates) and where A's entries are absent
@pytest.mark.parametrize("dtype", ["float32", "int32"])
@pytest.mark.parametrize("entries,absent", [(3, False), (200, False), (600, False), (600, True)])
def test_no_columns(b2, cuda, dtype, entries, absent):
    torch = cuda
    dt = getattr(torch, dtype)
    value = 1 if not absent else float("inf") if dtype == "float32" else 1073741823
    arp = torch.tensor([0, entries], dtype=torch.int64, device="cuda")
    aci = torch.zeros(entries, dtype=torch.int32, device="cuda")
    av = torch.full((entries,), value, dtype=dt, device="cuda")
    brp = torch.tensor([0, 1], dtype=torch.int64, device="cuda")
    b = (brp, torch.zeros(1, dtype=torch.int32, device="cuda"), torch.ones(1, dtype=dt, device="cuda"), 0)
    with pytest.raises(b2.B2Error) as e:
        b2.minplus_spgemm((arp, aci, av, 1), b)
    assert e.value.status == INVALID_INDEX
