"""capi._workspace: what is taken when the device has no room (no device needed)."""
import pytest


def test_the_least_is_taken_where_the_whole_does_not_fit(monkeypatch):
    import torch
    from vesper_b200 import capi
    asked, room = [], [100]

    def empty(n, dtype, device):
        asked.append(n)
        if n > room[0]:
            raise torch.cuda.OutOfMemoryError("full")
        return n

    monkeypatch.setattr(torch, "empty", empty)
    assert capi._workspace(50, "cpu", None, lambda a: a - 10, 30) == 50 and asked == [50]
    assert capi._workspace(500, "cpu", None, lambda a: a - 10, 30) == 20 and asked == [50, 500, 20]
    for least, args in ((None, None), (lambda a: a, 500)):
        with pytest.raises(torch.cuda.OutOfMemoryError):
            capi._workspace(500, "cpu", None, least, args)
    room[0] = 10
    with pytest.raises(torch.cuda.OutOfMemoryError):
        capi._workspace(500, "cpu", None, lambda a: a, 30)
