"""GPU time of the sparse product's row kernels against each other: no row class and no width of
the result falls off a cliff.  Bounds lie well between the measured ratio and that of the fault."""
import pytest

pytestmark = pytest.mark.gpu
ROWS = 1 << 16


def _ms(b2, torch, entries, each, columns):
    """Median time of a product of ROWS rows of `entries` x `each` candidates."""
    gen = torch.Generator(device="cuda").manual_seed(1)

    def matrix(length, cols):
        rp = torch.arange(ROWS + 1, dtype=torch.int64, device="cuda") * length
        ci = torch.randint(0, cols, (ROWS * length,), device="cuda", generator=gen, dtype=torch.int32)
        return rp, ci, torch.randint(0, 1000, (ROWS * length,), device="cuda", generator=gen, dtype=torch.int32), cols

    a, b = matrix(entries, ROWS), matrix(each, columns)
    times = []
    for _ in range(13):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        b2.minplus_spgemm(a, b)
        t1.record()
        torch.cuda.synchronize()
        times.append(t0.elapsed_time(t1))
    return sorted(times[3:])[5]


def test_rows_past_384_candidates(b2, cuda):
    """512 candidates against 384: 1.3, and 2.8 with the sorting network of 16 registers left rolled."""
    assert _ms(b2, cuda, 16, 32, ROWS) < 2.0 * _ms(b2, cuda, 16, 24, ROWS)


def test_rows_of_one_column(b2, cuda):
    """512 candidates in one column against distinct ones: 0.9, and 1.8 with a run walked by its head."""
    assert _ms(b2, cuda, 64, 8, 1) < 1.3 * _ms(b2, cuda, 64, 8, ROWS)


def test_one_long_row_of_a(b2, cuda):
    """One row of 2^20 entries against 2^13 rows of 128: 70, and 200 with eight lanes on the row."""
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(2)
    total = 1 << 20
    ones = torch.ones(total, dtype=torch.int32, device="cuda")
    b = (torch.arange(4097, dtype=torch.int64, device="cuda"), torch.arange(4096, dtype=torch.int32, device="cuda"),
         ones[:4096], 4096)
    ci = torch.randint(0, 4096, (total,), device="cuda", generator=gen, dtype=torch.int32)
    ms = {}
    for rows in (1, 1 << 13):
        a = (torch.arange(rows + 1, dtype=torch.int64, device="cuda") * (total // rows), ci, ones, 4096)
        times = []
        for _ in range(9):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            b2.minplus_spgemm(a, b)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        ms[rows] = sorted(times[3:])[3]
    assert ms[1] < 120 * ms[1 << 13], ms


def test_middling_rows_of_a_wide_result(b2, cuda):
    """2^13 rows of 3000 candidates in 150000 columns against 800000: 1.0, and 1.8 if accumulated densely."""
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(3)

    def matrix(rows, length, cols):
        return (torch.arange(rows + 1, dtype=torch.int64, device="cuda") * length,
                torch.randint(0, cols, (rows * length,), device="cuda", generator=gen, dtype=torch.int32),
                torch.randint(0, 1000, (rows * length,), device="cuda", generator=gen, dtype=torch.int32), cols)

    ms = {}
    a = matrix(1 << 13, 100, 1 << 14)
    for columns in (150000, 800000):
        b = matrix(1 << 14, 30, columns)
        times = []
        for _ in range(9):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            b2.minplus_spgemm(a, b)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        ms[columns] = sorted(times[3:])[3]
    assert ms[150000] < 1.4 * ms[800000], ms
