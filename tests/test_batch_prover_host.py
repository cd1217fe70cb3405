"""BatchFrameProver.prove joins the stream of the input MLEs on every way out, so that the
caller's tensors are free behind the launch stream; streams and launches stubbed."""
import pytest

from truepix_b200.frame import BatchFrameProver


class Stream:
    def __init__(self):
        self.waited_for = []

    def wait_stream(self, other):
        self.waited_for.append(other)


@pytest.mark.parametrize("refused", ["_input_mles", "_set_frames", "_rounds", None])
def test_the_mles_stream_is_joined(refused):
    p = object.__new__(BatchFrameProver)
    p.stream, p._mle_stream, p.groups, p.handle = Stream(), Stream(), {2: [0]}, None

    def call(name):
        def made(*args):
            if name == refused:
                raise RuntimeError(name)
            return 1
        return made

    for name in ("_input_mles", "_set_frames", "_rounds"):
        setattr(p, name, call(name))
    if refused:
        with pytest.raises(RuntimeError, match=refused):
            p.prove([None], [None], {2: None}, {2: None}, None)
    else:
        p.prove([None], [None], {2: None}, {2: None}, None)
        assert p.launches_last == 3
    assert p._mle_stream.waited_for == [p.stream]
    assert p.stream.waited_for == [p._mle_stream]
