"""Host-side shortcuts of a step: settings of the environment, workspace views."""
import torch

from tessweave_engine_b200.csrc.settings import setting
from tessweave_engine_b200.parts.base import Workspace


def test_settings_follow_the_environment(monkeypatch):
    monkeypatch.delenv("TESSWEAVE_PDL", raising=False)
    assert setting("TESSWEAVE_PDL") is None and setting("TESSWEAVE_PDL", "1") == "1"
    monkeypatch.setenv("TESSWEAVE_PDL", "0")
    assert setting("TESSWEAVE_PDL", "1") == "0"
    monkeypatch.setenv("TESSWEAVE_PDL", "")
    assert setting("TESSWEAVE_PDL", "1") == ""
    monkeypatch.setattr("os.environ", {"TESSWEAVE_PDL": "2"})       # another mapping in the environment's place
    assert setting("TESSWEAVE_PDL", "1") == "2" and setting("PATH") is None


def test_workspace_views_follow_their_buffers():
    ws = Workspace(torch.device("cpu"))
    a = ws.get("x", (2, 3), torch.float32)
    assert ws.get("x", (2, 3), torch.float32).data_ptr() == a.data_ptr() and ws.get("x", (3,), torch.float32).data_ptr() == a.data_ptr()
    big = ws.get("x", (5, 5), torch.float32)                        # grown: nobody gets the old one any more
    small = ws.get("x", (2, 3), torch.float32)
    assert small.data_ptr() == big.data_ptr() and small.shape == (2, 3)
    half = ws.get("x", (2, 3), torch.bfloat16)
    assert half.dtype == torch.bfloat16 and ws.get("x", (2, 3), torch.float32).dtype == torch.float32
    ws.prefix = "p."
    assert ws.get("x", (2, 3), torch.float32).data_ptr() != ws._buffers["x"].data_ptr()
    for n in range(1, 3 * Workspace.MAX_VIEWS):
        ws.get("y", (n,), torch.float32)
    assert len(ws._views) <= Workspace.MAX_VIEWS
    listed = ws.get("w", [2, 3], torch.float32)                     # a shape in a list, or a torch.Size
    assert listed.shape == (2, 3) and ws.get("w", listed.shape, torch.float32).data_ptr() == listed.data_ptr()
    zeros = ws.get("z", (4,), torch.int32, zero=True)
    assert int(zeros.sum()) == 0
