"""Which steps send a recurrence through the chunked kernels (parts/chunks.py): the rule against what both ways took, and the memory
it may ask for.  No GPU: the rule is arithmetic on a step's portions."""
import numpy as np
import pytest
import torch

from xyntetik_runner_b200 import kernels
from xyntetik_runner_b200.parts import chunks

# portions of a step, microseconds on one B200: the walk token by token, the chunks
MEASURED = [
    ("head", 8, 128, 128, [2048], 167, 74),
    ("head", 8, 128, 128, [800], 68, 59),
    ("head", 8, 128, 128, [640], 55, 55),
    ("head", 8, 128, 128, [680] * 3, 88, 77),
    ("head", 8, 128, 128, [1024] * 3, 130, 102),
    ("head", 8, 128, 128, [700] * 10, 226, 245),
    ("head", 8, 128, 128, [800] + [1] * 8, 103, 86),
    ("head", 8, 128, 128, [800] + [1] * 128, 110, 1002),
    ("head", 8, 128, 128, [2000] + [100] * 5, 255, 102),
    ("head", 8, 128, 256, [1500], 123, 95),
    ("head", 8, 128, 256, [800] + [1] * 8, 103, 163),
    ("head", 8, 128, 256, [800] + [1] * 128, 180, 2672),
    ("head", 8, 128, 256, [700] * 10, 364, 580),
    ("head", 32, 64, 64, [640], 41, 53),
    ("head", 32, 64, 64, [2048], 119, 94),
    ("head", 32, 64, 64, [700] * 10, 257, 334),
    ("key", 8, 128, 256, [2048], 222, 137),
    ("key", 8, 128, 256, [800], 96, 88),
    ("key", 8, 128, 256, [800] + [1] * 8, 130, 161),
    ("key", 8, 128, 256, [1600] + [1] * 128, 262, 2343),
    ("key", 8, 128, 256, [700] * 10, 440, 641),
    ("key", 8, 64, 64, [800], 62, 69),
    ("key", 8, 64, 64, [1600] + [1] * 8, 121, 74),
    ("mlstm", 8, 128, 256, [192], 106, 69),
    ("mlstm", 8, 128, 256, [2048], 912, 190),
    ("mlstm", 8, 128, 256, [200] * 3, 160, 92),
    ("mlstm", 8, 128, 256, [200] * 10, 226, 238),
    ("mlstm", 8, 128, 256, [200] + [1] * 32, 117, 278),
    ("mlstm", 8, 128, 256, [200] + [1] * 128, 162, 1361),
    ("mlstm", 8, 128, 256, [1600] + [1] * 8, 715, 209),
    ("mlstm", 32, 128, 128, [200] + [1] * 128, 251, 2755),
    ("mlstm", 32, 128, 128, [2048], 1182, 454),
    ("mlstm", 4, 128, 128, [300] * 3, 173, 76),
    ("mlstm", 4, 128, 128, [512] * 10, 296, 147),
]


class Step:
    def __init__(self, lens, dtype=torch.bfloat16):
        self.act_dtype, self.n, self.n_seg = dtype, sum(lens), len(lens)
        self.host = {"seg_len": np.array(lens, dtype=np.int32)}
        self.asked, self.memo = [], {}

    def once(self, key, make):
        if key not in self.memo:
            self.memo[key] = make()
        return self.memo[key]

    def buf(self, name, shape, dtype):
        self.asked.append(shape[0] * dtype.itemsize)
        return torch.empty(shape, dtype=dtype, device="meta")


@pytest.mark.parametrize("kind,H,D,V,lens,walk,in_chunks", MEASURED)
def test_the_faster_way_is_taken(kind, H, D, V, lens, walk, in_chunks):
    """Never a way that takes a seventh longer than the walk, and the chunks wherever they are a third faster."""
    taken = chunks.chunk_scratch(Step(lens), kind, H, D, V)
    if in_chunks > 1.15 * walk:
        assert taken is None
    if walk > 1.5 * in_chunks:
        assert taken is not None
    if taken is not None:
        assert taken.numel() >= kernels.chunked_floats(sum(lens), len(lens), H, D, V, kind) > 0


@pytest.mark.parametrize("kind", ["head", "key", "mlstm"])
@pytest.mark.parametrize("lens", [[7937] + [1] * 255, [2048] * 40, [65536], [40000, 3], [3000] * 3])
def test_scratch_is_bounded(kind, lens):
    """The walk needs no memory beside the states: a step that it can take never asks for more than MOST_BYTES for the other way."""
    for H, D, V in ((8, 128, 256), (32, 128, 256), (4, 64, 64)):
        step = Step(lens)
        chunks.chunk_scratch(step, kind, H, D, V)
        assert sum(step.asked) <= 1 << 28
        assert chunks.chunk_scratch(Step(lens, torch.float32), kind, H, D, V) is None
