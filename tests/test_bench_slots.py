"""The byte model of the solver's cycle with the matrix in slot form: as with
CSR (test_bench_models.py) but for the matrix, which every one of the 2 l
products reads once."""
import bench


def test_cycle_bytes_with_slots():
    n, nnz = 1000, 4900
    for l in (1, 2, 4):
        csr, five, seven = (bench.bicgstabl_cycle_bytes(n, nnz, l, slots=s) for s in (0, 5, 7))
        assert csr - five == 2 * l * (12 * nnz + 4 * (n + 1) - 41 * n)
        assert seven - five == 2 * l * 16 * n
        assert bench.bicgstabl_cycle_bytes(n, nnz, l, slots=3) == five
