"""The first call of a storage on a caller's stream: what the storage prepared
on its own stream is in place, whatever that stream still has to do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_call_on_another_stream(pkg, orc):
    torch = pytest.importorskip("torch")
    t = np.random.default_rng(5).integers(2, 6, size=300_000).astype(np.uint8)
    want = orc.sa_bwt(t)
    d = torch.from_numpy(t).cuda()
    torch.cuda.synchronize()
    for _ in range(20):
        s = torch.cuda.Stream()
        with pkg.Storage(0) as st:
            st.set_stream(s.cuda_stream)
            o = torch.empty_like(d)
            s.synchronize()
            st.pfp_bwt_device(d.data_ptr(), o.data_ptr(), len(t))
            assert np.array_equal(o.cpu().numpy(), want)
