"""Programs that step call by call: the waveform and phase tables go through a
ring of slots per stream, which must hold every value until its kernels have
read it however many calls are queued, on whichever stream."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = 150  # more than twice round the ring


def _scene(fd):
    g = fd.Grid((40, 36, 1), grid_spacing=155e-9)
    g[0:5, :, :] = fd.PML()
    g[:, -5:, :] = fd.PML()
    g[20, 8:28, 0] = fd.LineSource(period=11)
    g[12, 9, 0] = fd.PointSource(period=7, pulse=True)
    g[:, 18, 0] = fd.LineDetector(name="line")
    g[:, 10, :] = fd.DFTPlaneDetector(frequencies=[1.0 / (11 * g.time_step), 1.0 / (8 * g.time_step)], name="dft")
    return g


def _results(g):
    torch.cuda.synchronize()
    return [g.E.cpu(), g.H.cpu(), g.line.E.tensor().cpu(), g.line.H.tensor().cpu(),
            torch.view_as_real(g.dft.dft.cpu())]


@pytest.mark.parametrize("how", ["step", "halves", "streams", "long_tables"])
@pytest.mark.parametrize("prec", ["float64", "float32"])
def test_calls_in_any_number_equal_one_run(fd, prec, how):
    fd.set_backend("gb300." + prec)
    one = _scene(fd)
    one._ensure_engine().set_tuning(persistent=1)
    one.run(STEPS, progress_bar=False)
    g = _scene(fd)
    g._ensure_engine().set_tuning(persistent=1)
    streams = [torch.cuda.Stream() for _ in range(6)]  # more than the stager keeps rings for
    torch.cuda.synchronize()
    done = 0
    while done < STEPS:
        if how == "halves":
            g.update_E()
            g.update_H()
            g.time_steps_passed += 1
            done += 1
        elif how == "streams":
            s, last = streams[done % 6], streams[(done - 1) % 6]
            s.wait_stream(last)
            with torch.cuda.stream(s):
                g.step()
            done += 1
        elif how == "long_tables":
            n = min(1 if done % 3 else 50, STEPS - done)
            g.run(n, progress_bar=False)
            done += n
        else:
            g.step()
            done += 1
    for a, b in zip(_results(one), _results(g)):
        assert np.array_equal(a.numpy(), b.numpy())
