"""Stream handles as the binding passes them to the library (no GPU)."""
import pytest

from marigold_b200 import _lib


class _Library:
    def __init__(self):
        self.streams = []

    def mgbvh_set_stream(self, ptr, stream):
        self.streams.append(stream.value)
        return 0


@pytest.mark.parametrize("handle,passed", [(None, None), (0, 1), (1, 1), (0x7F00, 0x7F00)])
def test_default_stream_is_passed_by_name(handle, passed):
    """Handle 0 is torch's default stream, which a context's calls wait for:
    it must not reach the library as NULL, its own stream ordered after no other."""
    ctx = _lib.Context.__new__(_lib.Context)
    ctx.L, ctx.ptr = _Library(), None
    ctx.set_stream(handle)
    assert ctx.L.streams == [passed]
