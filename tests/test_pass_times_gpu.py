"""What the calls report as device time."""
import pytest

import gguf_util as gu

pytestmark = pytest.mark.gpu


def test_the_time_of_a_pass_leaves_capturing_out(ctx, pkg, tmp_path):
    """The second pass of a kind is captured, which takes the host milliseconds; the device time that the call reports is the pass's."""
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=2, extra=["--layers", 24])
    m = pkg.Model(ctx, path, 64)
    m.verify([1, 2, 3], 0)
    for tokens in ([1, 2, 3, 4, 5], [5] * 9, [7] * 16):
        ms = [m.verify(tokens, 0)[1] for _ in range(6)]
        assert ms[1] < 2 * max(ms[2:]) + 0.5, ms           # (2.3 ms with it)
    b = pkg.Batch(m, 20, 32)
    ms = [b.step([3] * 20, list(range(20)), [4] * 20)[1] for _ in range(6)]
    assert ms[1] < 2 * max(ms[2:]) + 0.5, ms
    b.free(); m.free()
