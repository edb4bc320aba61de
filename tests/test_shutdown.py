"""The end of a process winds everything up, whatever the session has to report when it closes."""
import types

import pytest

from autodist_b200.autodist import AutoDist


def test_a_session_that_raises_does_not_keep_the_coordinator_waiting():
    joined = []

    def close():
        raise RuntimeError("a lookup met an id outside its table")
    job = types.SimpleNamespace(_session=types.SimpleNamespace(close=close), _coordinator=types.SimpleNamespace(join=lambda timeout: joined.append(timeout)))
    with pytest.raises(RuntimeError, match="outside its table"):
        AutoDist._shutdown(job)
    assert joined == [30]
