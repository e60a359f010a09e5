"""The footprint estimate counts what a handle keeps between calls: padded
copies of the factors for a rank that is no vector multiple, and the per-CTA
copies of short outputs."""
import alto_b200 as ab
from alto_b200 import serve
from test_serve_host import _req


def test_footprint_counts_padded_copies():
    dims = (5_000_000, 4_000_000, 3_000_000)
    for kind in (serve.ALS, serve.APR):
        for ftype, size, vec in ((ab.F32, 4, 4), (ab.F64, 8, 2)):
            whole, odd = (serve.footprint(_req(kind, dims, 20_000_000, r, ftype)) for r in (32, 33))
            # one more column of the model (two to four copies of it) and of the nonzeros' rows, and the padded copies
            grown = sum(dims) * size * 5 + 20_000_000 * size + (33**2 - 32**2) * 8 * 6
            assert odd - whole <= grown + sum(dims) * (32 + vec) * size
            assert odd >= whole + sum(dims) * (32 + vec) * size * 0.6


def test_footprint_counts_short_output_copies():
    small, large = (serve.footprint(_req(serve.APR, (300, 200, 100), n, 16)) for n in (1_000_000, 2_000_000))
    # key, value, order, stream and rows of a nonzero, and 32 bytes of copies up to 48 MB
    per = 8 + 4 + 4 * 3 + 16 * 4 + 3 * (8 + 4) + 24
    assert large - small >= 1_000_000 * per + (16 << 20)
