"""The tcgen05 kernels and the choice between the staged kernels at the sizes where they can go wrong, against the integer
kernel, bit for bit: halves of a tile without columns, rows and columns that end inside a tile, one k-tile and more k-tiles
than stages, chains that end inside and at the end of K, K slices, operands that 16-byte loads cannot read, output dtypes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PAIRS = (("e4m3", "e4m3"), ("e5m2", "e4m3"), ("e4m3", "e5m2"))


def codes(rng, rows, K, fmt):
    """Codes around the middle of the exponent range, 1 % of any value, two non-finite ones."""
    x = rng.integers(0x28, 0x58, (rows, K), dtype=np.uint8) | (rng.integers(0, 2, (rows, K), dtype=np.uint8) << 7)
    x = np.where(rng.random((rows, K)) < 0.01, rng.integers(0, 256, (rows, K), dtype=np.uint8), x)
    top = 0x7F if fmt == "e4m3" else 0x7C
    x = np.where((x & 0x7F) >= top, 0x38, x).astype(np.uint8)
    x[rows // 2, K // 2] = 0x7F
    if fmt == "e5m2":
        x[rows // 3, K // 3] = 0xFC
    return x


def same(fn, *args, **kw):
    import gpu_runner
    run = getattr(gpu_runner, fn)
    got, want = run(*args, kernel="staged", **kw), run(*args, kernel="integer", **kw)
    bad = np.argwhere(got != want)
    assert bad.size == 0, f"{len(bad)} of {got.size} differ, first {bad[0]}: {got[tuple(bad[0])]:#x} != {want[tuple(bad[0])]:#x}"


@pytest.mark.parametrize("fast", (True, False), ids=("fast", "slow"))
@pytest.mark.parametrize("preset", (16, 32))
@pytest.mark.parametrize("fmts", PAIRS, ids="x".join)
@pytest.mark.parametrize("M,N,K", ((1, 1, 16), (128, 64, 32), (129, 65, 176), (257, 200, 528),
                                   (1160, 2064, 16), (1160, 2064, 144), (1160, 2192, 272)))
def test_tiles(M, N, K, fmts, preset, fast):
    """The last three have 170 and 180 tiles of 128 columns (two waves) and 90 of 256 columns (one): both tile widths run,
    the mixed pairs with 32 products per block on the narrow one; 2064 = 8 x 256 + 16 leaves a tile with one half."""
    rng = np.random.default_rng(M + N + K + preset)
    same("accumulate", codes(rng, M, K, fmts[0]), codes(rng, N, K, fmts[1]), fmt_a=fmts[0], fmt_b=fmts[1], preset=preset, fast=fast)


@pytest.mark.parametrize("out", ("float32", "bfloat16", "float16", "float8_e4m3fn", "float8_e5m2"))
@pytest.mark.parametrize("M,N,K", ((130, 208, 160), (1160, 2064, 160)))
@pytest.mark.parametrize("fast", (True, False), ids=("fast", "slow"))
def test_output_stage(M, N, K, out, fast):
    rng = np.random.default_rng(5)
    same("scaled_mm", codes(rng, M, K, "e4m3"), codes(rng, N, K, "e4m3"), 0.37, 2.5, out=out, preset=32, fast=fast,
         **({"scale_result": 0.125} if out.startswith("float8") else {}))


@pytest.mark.parametrize("plan", ((16, False, 1, "none"), (32, False, 1, "none"), (16, True, 3, "serial"), (16, False, 5, "pairwise"),
                                  (32, True, 4, "contiguous"), (32, False, 3, "contiguous"), (32, True, 8, "contiguous")),
                         ids=lambda p: f"nfma{p[0]}-{'fast' if p[1] else 'slow'}-S{p[2]}-{p[3]}")
@pytest.mark.parametrize("fmts", PAIRS, ids="x".join)
def test_slices(fmts, plan):
    """K slices on tcgen05 (and, with more splits than k-tiles, the general walkers)."""
    preset, fast, S, scheme = plan
    rng = np.random.default_rng(S + preset)
    for M, N, K in ((70, 90, 272), (200, 130, 2064), (40, 300, 16)):
        same("accumulate", codes(rng, M, K, fmts[0]), codes(rng, N, K, fmts[1]), fmt_a=fmts[0], fmt_b=fmts[1], preset=preset,
             fast=fast, S=S, scheme=scheme)


@pytest.mark.parametrize("fast", (True, False), ids=("fast", "slow"))
@pytest.mark.parametrize("fmts", PAIRS + (("e5m2", "e5m2"),), ids="x".join)
@pytest.mark.parametrize("M,N,K", ((3, 5, 1), (16, 130, 37), (150, 129, 401), (65, 66, 2001)))
def test_operands_without_16_byte_loads(M, N, K, fmts, fast):
    rng = np.random.default_rng(K)
    for preset in (16, 32):
        same("accumulate", codes(rng, M, K, fmts[0]), codes(rng, N, K, fmts[1]), fmt_a=fmts[0], fmt_b=fmts[1], preset=preset,
             fast=fast)


@pytest.mark.parametrize("kernel", ("staged", "staged-rows"))
@pytest.mark.parametrize("ld_pad", (1, 8, 16))
@pytest.mark.parametrize("M,N,K", ((16, 130, 48), (150, 129, 416)))
def test_odd_leading_dimensions(M, N, K, ld_pad, kernel):
    """K a multiple of 16 but rows that start anywhere (ld_pad 16: the 16-byte loads of the same call)."""
    import gpu_runner
    rng = np.random.default_rng(K + ld_pad)
    a, b = codes(rng, M, K, "e5m2"), codes(rng, N, K, "e4m3")
    for fast in (True, False):
        got, want = (gpu_runner.scaled_mm(a, b, 0.37, 2.5, fmt_a="e5m2", out="float32", preset=32, fast=fast, kernel=k, ld_pad=ld_pad)
                     for k in (kernel, "integer"))
        assert np.array_equal(got, want)
