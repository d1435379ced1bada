"""sdbe_resample_chunks on at most two chunks per SM (no pipeline): the same
floats as among more chunks, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trim", [0, 150, 240])
def test_few_chunks_equal_many(trim):
    import __graft_entry__ as g

    g.build()
    import torch

    from sdbe_gb300 import Resampler, _native as N

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = torch.randn(2 * sms + 1, 36608, device="cuda", generator=torch.Generator(device="cuda").manual_seed(trim))
    out = torch.empty(2 * sms + 1, 32768, device="cuda")

    def run(lo, hi):
        out[lo:hi].zero_()
        torch.cuda.synchronize()
        N.check(N.lib().sdbe_resample_chunks(r.handle, x[lo:hi].data_ptr(), hi - lo, out[lo:hi].data_ptr(), None), r.handle)
        r.sync()
        return out[lo:hi].clone()

    with Resampler(trim_mhz=trim, max_frames=1) as r:
        ref = run(0, 2 * sms + 1)
        for lo, hi in ((0, 1), (3, 5), (0, sms - 1), (1, sms + 1), (0, sms + 1), (1, 2 * sms + 1)):
            assert torch.equal(run(lo, hi), ref[lo:hi]), (lo, hi)
