"""The division and root of the walks' draws over every word they can meet."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_division_and_root_of_all_words_are_correctly_rounded():
    from nozomi_b200 import _lib as L
    differ = torch.ones(1, dtype=torch.int64, device="cuda")
    L.check(L.load().nz_probe_draw_operators(differ.data_ptr(), None), "nz_probe_draw_operators")
    torch.cuda.synchronize()
    assert int(differ.item()) == 0
