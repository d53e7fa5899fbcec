"""Training operator with its [M, H] matrices held for a part of the tokens at a time: the 64-bit reference
and bounds of ``test_pair_train_gpu`` on calls of two to five chunks, with overflowed rows in each, next to a
guard region that no launch may touch."""
import pytest
import torch

from sparser_faster_llms_b200 import _lib
from test_pair_train_gpu import ops, run_case  # noqa: F401  (ops: the module's fixture)

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
GUARD = 32 << 20


@pytest.fixture
def chunked(monkeypatch):
    """Sends the operator's calls through the chunked entry points; returns what they were given."""
    seen, plain = [], _lib.call

    def start(max_rows):
        def call(fn, device, *args):
            if not fn.startswith("b200_hybrid_train_"):
                return plain(fn, device, *args)
            m, d, h, _, tail = args[12:17]
            need = _lib.load_library().b200_hybrid_train_scratch_bytes_chunked(
                m, d, h, tail, int(fn.endswith("backward")), max_rows)
            scratch = torch.full((need + GUARD,), 0x5A, dtype=torch.uint8, device=DEV)
            plain(fn + "_chunked", device, *args[:-2], scratch.data_ptr(), need, max_rows)
            seen.append(scratch[need:])
        monkeypatch.setattr(_lib, "call", call)
        return seen
    return start


@pytest.mark.parametrize("m,d,h,max_rows,hot", [
    (999, 1024, 4096, 256, 0), (1300, 256, 2048, 512, 0), (300, 768, 1280, 1, 0),
    (700, 512, 2048, 256, 9), (9000, 512, 1280, 4096, 0)])  # the last: carried sums of tiles cut along k
def test_chunks_of_a_step(chunked, m, d, h, max_rows, hot):
    seen = chunked(max_rows)
    taken, left = run_case(m, d, h, 0.03, hot=hot)
    assert len(seen) == 2 and all(bool((s == 0x5A).all()) for s in seen)
    if hot:
        assert taken == (m + hot - 1) // hot and left == 0


def test_one_chunk_is_the_plain_call(chunked):
    seen = chunked(4096)
    run_case(700, 512, 2048, 0.03, hot=9)
    assert len(seen) == 2 and all(bool((s == 0x5A).all()) for s in seen)
