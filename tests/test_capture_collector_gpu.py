"""No garbage is collected while a decode graph is captured: a dead runner's graphs given back then spoil the capture."""
import gc

import pytest
import torch

import test_tadinex as T

pytestmark = pytest.mark.gpu


def test_collector_waits_for_the_capture(monkeypatch):
    from uniserve_v1_b200.engine.runner import CausalLmRunner
    seen, body = [], CausalLmRunner._decode_body

    def watched(self, *a, **kw):
        seen.append((torch.cuda.is_current_stream_capturing(), gc.isenabled()))
        return body(self, *a, **kw)
    monkeypatch.setattr(CausalLmRunner, "_decode_body", watched)
    form = ("cuda", torch.float32)
    c, w, model = T.build("odd", form)
    T.run(T.engine(model), "a", T.ids(c, 5, 2, w, form), [3, 1, 1])
    assert (True, False) in seen and (True, True) not in seen and gc.isenabled()
