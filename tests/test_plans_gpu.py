"""Which kernel a call takes, by the geometry that the library reports for it (masked calls, aligned rows)."""
import pytest

from flintnsteel_b200.sampler import BF16, F32, Sampler

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

V = 151_936


@pytest.mark.parametrize("k_cap, longest, longest_large", [(64, 4136, 636), (128, 3816, 316)])
@pytest.mark.parametrize("rows", [1, 8, 12])
def test_small_batches_take_the_cluster_kernel(rows, k_cap, longest, longest_large):
    """Sixteen CTAs per row up to the longest history that the kernel's 112 KB have room for: with k_cap 64 that covers the
    4,096 ids of a default handle."""
    s = Sampler(0, max_rows=12, max_vocab=262_144, k_cap=k_cap)
    for dtype, vocab, strides in ((F32, V, (0, 8, 2048, longest - 40, longest)), (BF16, V, (0, 2048, 4096)),
                                  (F32, 262_144, (0, longest_large))):
        for stride in strides:
            p = s.plan(dtype, vocab, rows, stride)
            assert p["slices"] == 16 and p["slice_len"] == -(-vocab // 16 // 128) * 128, (dtype, vocab, stride, p)
    s.close()
