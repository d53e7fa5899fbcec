"""Sizes of the scratch that calls on the paired tensor-core GEMM ask for, against what each of their
launches writes.  A launch cuts its last wave of tiles along k, and how depends on the number of tiles,
so every row chunk of a call is looked at by itself.  The library sizes for 148 SMs without a device."""
import ctypes
import random

import pytest

from sparser_faster_llms_b200 import _lib, build

PAIRS, TILE, STAGE_K, CUT_KSTEPS = 74, 256, 64, 64
SHAPES = [(1024, 4096), (2048, 5632), (2048, 8192), (2048, 11008), (4096, 11008), (4096, 16384)]


@pytest.fixture(scope="module")
def lib():
    build.build_library()
    return _lib.load_library()


def range_bytes(tiles, k, own_kernel):
    """fp32 sums of the ranges that a product of `tiles` tiles is cut into."""
    ksteps, tail = -(-k // STAGE_K), tiles % PAIRS
    own_kernel = own_kernel and tiles < PAIRS
    if tail == 0 or (not own_kernel and ksteps < CUT_KSTEPS):
        return 0
    most = 8 if own_kernel else 4
    splits = min(PAIRS // tail, ksteps // 4, most)
    return 0 if splits < 2 else tail * splits * TILE * TILE * 4


def chunks(m, h, terms, max_rows):
    rows = (1 << 30) // (h * 2 * terms) // TILE * TILE
    if max_rows:
        rows = min(rows, max(TILE, max_rows // TILE * TILE))
    rows = min(m, rows)
    return [min(rows, m - r) for r in range(0, m, rows)]


def one_sm_tiles(m, d, h):
    """Whether a gated bf16 call runs on one-SM tiles: its line, and one wave of them."""
    start = 33 if d * h <= 12 << 20 else 40 if d * h <= 1 << 24 else 80
    return start <= m <= 512 and -(-m // 128) * h // 128 <= 148 and not (m <= 128 and 132 < h // 64 <= 148)


def mlp_need(m, d, h, terms, max_rows, cf=2):
    if terms == 3 and not 0 < max_rows < m and m * d * h < 1 << 36:
        return m * h // cf * 4  # fp32 hidden values in the slots of the slabs
    if terms == 1 and not 0 < max_rows < m and one_sm_tiles(m, d, h):
        return m * h * 2
    sizes = chunks(m, h, terms, max_rows)
    cut = 0
    for rows in set(sizes):
        mt = -(-rows // TILE)
        cut = max(cut, range_bytes(mt * (h // TILE), d, False),
                  range_bytes(mt * (d // TILE), h * terms, True))
    return 240 + sizes[0] * h * 2 * terms + 256 + cut  # 240: from 16-byte to 256-byte alignment


def token_counts(h, terms):
    rnd = random.Random(h + terms)
    chunk = (1 << 30) // (h * 2 * terms) // TILE * TILE
    edges = [k * chunk + e for k in (1, 2) for e in (-1, 0, 1, 100, 256, 777, 1024)]
    return edges + [rnd.randint(64, 3 * chunk) for _ in range(60)]


@pytest.mark.parametrize("d,h", SHAPES)
@pytest.mark.parametrize("gated,flags", [(1, 0), (1, _lib.FLAG_HIGH_PRECISION), (0, 0)])
def test_fused_mlp_scratch_holds_every_chunk(lib, d, h, gated, flags):
    terms = 3 if flags else 1
    seen = 0
    for m in token_counts(h, terms):
        got = lib.b200_twell_mlp_scratch_bytes(m, d, h, gated, flags)
        need = mlp_need(m, d, h, terms, 0)
        assert got == 0 or need <= got <= need + 256, m
        seen += got > 0
    assert seen > 40


@pytest.mark.parametrize("cf", [2, 4, 8])
def test_high_precision_scratch_follows_the_compression_factor(lib, cf):
    flags = _lib.FLAG_HIGH_PRECISION | _lib.scratch_cf(cf)
    for m, d, h in ((777, 2048, 8192), (100, 1024, 4096), (16383, 1024, 4096)):
        assert lib.b200_twell_mlp_scratch_bytes(m, d, h, 1, flags) == m * h // cf * 4
    for m, d, h in ((40, 1024, 4096), (100, 2048, 8192)):  # bf16 on one-SM tiles: hidden values, no sums
        assert lib.b200_twell_mlp_scratch_bytes(m, d, h, 1, _lib.scratch_cf(cf)) == 2 * m * h


@pytest.mark.parametrize("max_rows", [1, 256, 600, 4096])
def test_chunked_scratch_holds_every_chunk(lib, max_rows):
    for d, h in SHAPES:
        for m in (320, 700, 1000, 5000, 70000):
            got = lib.b200_twell_mlp_scratch_bytes_chunked(m, d, h, 1, 0, max_rows)
            assert got == 0 or got >= mlp_need(m, d, h, 1, max_rows), (m, d, h)
            assert got <= lib.b200_twell_mlp_scratch_bytes(m, d, h, 1, 0) + (1 << 26)


def train_need(m, d, h, tail, bwd, max_rows):
    sizes = chunks(m, h, 1, max_rows)
    nt, mt = h // TILE, lambda rows: -(-rows // TILE)
    cut = 0 if bwd else range_bytes(mt(m) * nt, d, False)
    for rows in set(sizes):
        cut = max(cut, range_bytes(mt(rows) * nt, d, False),
                  range_bytes(mt(rows) * (d // TILE), (2 if bwd else 1) * h, True),
                  range_bytes(3 * nt * (d // TILE), rows, False) if bwd else 0)
    rows_out = tail * (4 + 2 * d + (4 if bwd else 2) * h) + m * 9
    carry = 12 * h * d if bwd and len(sizes) > 1 else 0
    return rows_out + sizes[0] * h * (6 if bwd else 2) + cut + carry + \
        (0 if bwd else mt(m) * nt * 64)


@pytest.mark.parametrize("d,h", SHAPES + [(256, 256)])
@pytest.mark.parametrize("bwd", [0, 1])
def test_training_scratch_holds_every_chunk_and_stays_bounded(lib, d, h, bwd):
    for max_rows in (0, 256, 5000):
        for m in token_counts(h, 1)[::3] + [1, 129, 5_000_000]:
            for tail in (0, min(m, 2048)):
                got = lib.b200_hybrid_train_scratch_bytes_chunked(m, d, h, tail, bwd, max_rows)
                need = train_need(m, d, h, tail, bwd, max_rows)
                assert need <= got <= need + (1 << 14)
    # a step of five million tokens: bounded matrices and a few bytes per token
    most = (3 if bwd else 1) * (1 << 30) + 12 * h * d + 5_000_000 * (9 + h / 4) + (1 << 28)
    assert lib.b200_hybrid_train_scratch_bytes(5_000_000, d, h, 2048, bwd) < most


def test_training_takes_as_many_tokens_as_the_other_entry_points(lib):
    buf = (ctypes.c_char * 512)()
    p = (ctypes.addressof(buf) + 255) & ~255
    for m, status in ((1 << 27, -6), (1 << 30, -6), ((1 << 30) + 1, -4)):
        # a valid call but for its scratch (no CUDA call is made), or one token too many
        assert lib.b200_hybrid_train_forward(*[p] * 12, m, 256, 256, 8, 0, None, 0, p, 64, None) == status
        assert lib.b200_hybrid_train_backward(*[p] * 12, m, 256, 256, 8, 0, None, 0, p, 64, None) == status
