"""That steps really are launched before the host has seen the lists of the step in front, and launched anew where a hypothesis has ended: launches of the kernel
that runs a step's layers, steps, and the bytes that the lists take on their way to the host (16 an entry with the tags that tell the host when it is new, 12
without)."""
import ctypes

import pytest

from tests.test_gpu_step_ahead import _batch, _bits, _net

pytestmark = pytest.mark.gpu


def _run(net, cfg, batch, beam, width, ahead, data):
    from marian_dev_b200 import decoder
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=width, max_steps=int(1.5 * width) + 2)
    stepper.set_option("step_ahead", ahead)
    search = decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper)
    first = search.search(*data)
    stepper.search_stats(reset=True)
    search.d2h_bytes = 0
    check(lib().mi8_kernel_times_begin())
    try:
        out = search.search(*data)
    finally:
        records, n = (Mi8KernelTime * 64)(), ctypes.c_int(0)
        check(lib().mi8_kernel_times_end(records, 64, ctypes.byref(n)))
    assert _bits([first]) == _bits([out])
    launches = sum(r.launches for r in records[:n.value] if "decoder_rows_kernel" in r.name.decode())
    return _bits([out]), launches, stepper.search_stats()["steps"], search.d2h_bytes


@pytest.mark.parametrize("dim,batch,beam,eos_bias", [(256, 1, 1, -50.0), (256, 8, 4, -50.0), (512, 16, 1, -50.0), (256, 8, 4, 3.0), (256, 32, 1, 2.5), (512, 4, 4, 3.0)])
def test_used(cuda_device, dim, batch, beam, eos_bias):
    from marian_dev_b200 import ops
    cfg, net = _net(cuda_device, dim, 1003, eos_bias, dim + batch)
    data = _batch(cfg, batch, 11, 3)
    got, launches, steps, down = _run(net, cfg, batch, beam, 11, 1, data)
    want, plain_launches, plain_steps, plain_down = _run(net, cfg, batch, beam, 11, 0, data)
    assert got == want and steps == plain_steps == plain_launches and ops.poll_status() == 0
    if eos_bias < 0:                # no hypothesis ends in front of the last step: every step but the first was launched ahead and stood
        assert launches == steps and 12 * down == 16 * plain_down
        assert plain_down == 12 * batch * beam * steps
    else:                           # steps were launched ahead, and some of them were launched anew
        assert launches > steps and down > plain_down
