"""The bench's unique bytes of the padded inverse passes, counted launch by
launch: a buffer that two operands of one launch read counts once."""
import bench


def _launch_bytes(reads, writes, size):
    return sum(size[b[0]] for b in set(reads)) + sum(size[b[0]] for b in writes)


def test_inverse_pass_bytes():
    for n, pb in ((64, 8), (512, 4)):
        M, Kz, cs = 3 * n // 2, n // 2 + 1, 2 * pb
        # k-space grid, compact rows (x padded), padded rows (x and y padded)
        size = {"f": n * n * Kz * cs, "c": M * n * Kz * cs, "p": M * M * Kz * cs}
        xinv = yinv = 0
        for _ in ("phi", "phi2"):  # the six Hessians of a field
            # of f: f, i g_x f and -g_x^2 f
            xinv += _launch_bytes([("f",)] * 3, [("c", k) for k in range(3)], size)
            yinv += _launch_bytes([("c", 2), ("c", 1), ("c", 0)], [("p", k) for k in range(3)], size)
            yinv += _launch_bytes([("c", 1), ("c", 0), ("c", 0)], [("p", k) for k in range(3)], size)
        for _ in range(5):  # the pair products of the third order
            yinv += _launch_bytes([("c", 0)], [("p", 0)], size)
        b = bench.algorithmic_bytes_ic(n, pb)
        assert b["conv_xinv"] == xinv
        assert b["conv_yinv"] == yinv
