"""The quantiser kernel multiplies by rounded reciprocals where the reference's fp16 ops divide
(csrc/w4a16_quantize.cu): the integers are the same for every pair of values that can meet, checked over all of them."""
import torch


def _halves(lo, hi):
    """All fp16 values with bit patterns lo .. hi."""
    return torch.arange(lo, hi + 1, dtype=torch.int32).to(torch.int16).view(torch.float16)


def _scales():
    low = torch.tensor([1e-5]).half()
    d = torch.cat((_halves(int(low.view(torch.int16)), 0x7bff), torch.tensor([float("inf")]).half())).float()
    return d, (d / 15.0).half()


def test_scale_by_reciprocal_of_fifteen():
    d, scale = _scales()
    assert torch.equal((d * torch.tensor(1.0 / 15.0, dtype=torch.float32)).half(), scale)


def test_code_by_reciprocal_of_the_scale():
    """rint(fp16(w * rn(1 / s))) == rint(fp16(w / s)) for every finite fp16 w and every scale the quantiser can produce, where
    the integer matters: beyond 512 both only have to stay beyond every clamp.  (Negative w: both sides change sign.)"""
    scales = torch.unique(_scales()[1].float())
    scales = scales[torch.isfinite(scales)]
    w = _halves(0, 0x7bff).float()
    assert scales.numel() > 20000
    for part in scales.split(128):
        s = part[:, None]
        old = torch.round((w / s).half().float())
        new = torch.round((w * (1.0 / s)).half().float())
        bad = (old != new) & ((old < 512) | (new < 512))
        assert not bool(bad.any()), (part[bad.any(1)][:3], w[bad.any(0)][:3])
