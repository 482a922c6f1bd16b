"""Plans and batches made from CUDA weights whose values the current torch stream
has yet to write: they hold the values, not what the memory held before."""
import numpy as np
import pytest

from conftest import crandn
from openvsip_b200 import Fastconv, replica_spectrum
from openvsip_b200.batch import Batch

pytestmark = pytest.mark.gpu
RTOL = 2e-6  # the suite's bound for single-precision transforms


def _late(values, delay=40_000_000):
    """A tensor that becomes `values` after some 20 ms of queued work."""
    import torch
    src = torch.from_numpy(values).cuda()
    dst = torch.zeros_like(src)
    torch.cuda.synchronize()
    torch.cuda._sleep(delay)
    dst.copy_(src)
    return dst


@pytest.mark.parametrize("side", [False, True])  # the default stream, a stream of the program's own
@pytest.mark.parametrize("n,weight_rows", [(512, 1), (512, 4), (480, 1), (1072, 4)])
def test_plan_made_while_its_weights_are_written(oracle, n, weight_rows, side):
    import torch
    rng = np.random.default_rng(n)
    x, w = crandn(rng, (4, n)), crandn(rng, (weight_rows, n) if weight_rows > 1 else (n,))
    with torch.cuda.stream(torch.cuda.Stream() if side else torch.cuda.current_stream()):
        y = Fastconv(_late(w), 4)(torch.from_numpy(x).cuda()).cpu().numpy()
    want = np.fft.ifft(np.fft.fft(x.astype(np.complex128)) * w.astype(np.complex128))
    assert oracle.rel_l2(y, want) <= RTOL


def test_batch_replica_and_spectrum_made_while_written(oracle):
    import torch
    rng = np.random.default_rng(3)
    x, r = crandn(rng, (4, 512)), crandn(rng, (512,))
    spec = np.fft.fft(r.astype(np.complex128))
    assert oracle.rel_l2(replica_spectrum(_late(r), matched=False).cpu().numpy(), spec) <= RTOL
    b = Batch()
    rid = b.add_replica(_late(r), kind="time")
    dx = torch.from_numpy(x).cuda()
    out = torch.zeros_like(dx)
    b.set_jobs([(dx, out, rid)])
    torch.cuda.synchronize()
    b.run()
    b.sync()
    assert oracle.rel_l2(out.cpu().numpy(), np.fft.ifft(np.fft.fft(x.astype(np.complex128)) * spec)) <= RTOL
