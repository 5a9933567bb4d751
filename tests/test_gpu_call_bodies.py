"""What the host bodies of the ops keep, hold and share: the answer about a weight zero point, the interpreter lock, errors raised inside a call,
scratch on several streams."""
import threading
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(a, dev):
    return torch.from_numpy(np.array(a)).to(dev)


def _conv_case(ops, orc, dev, seed=0):
    """(call(w_zero_point tensor), want(zero points)) of a small QLinearConv."""
    rng = np.random.default_rng(seed)
    x, w = rng.integers(0, 256, (2, 24, 9, 10), dtype=np.uint8), rng.integers(-127, 128, (16, 24, 3, 3)).astype(np.int8)
    ws = rng.uniform(0.001, 0.002, 16).astype(np.float32)
    xt, wt, wst = _t(x, dev), _t(w, dev), _t(ws, dev)

    def call(wz):
        return ops.QLinearConv(xt, 0.02, np.uint8(5), wt, wst, wz, 0.05, np.uint8(100), strides=(1, 1), pads=(1, 1)).cpu().numpy()

    def want(wz):
        return orc.requantize(orc.conv_integer(x, w, 5, wz, (1, 1), (1, 1)), 0.02, ws, 0.05, 100, channel_axis=1)

    return call, want


def test_weight_zero_points_changed_in_place(ops, orc, dev):
    """A zero-point tensor that was all zeros and is changed in place: ordinary tensors, and inference tensors, which have no version counter."""
    call, want = _conv_case(ops, orc, dev)
    zero, other = want(np.zeros(16, np.int8)), want(np.full(16, 3, np.int8))
    assert (zero != other).any()
    for inference in (False, True):
        with torch.inference_mode(inference):
            wz = torch.zeros(16, dtype=torch.int8, device=dev)
            assert wz.is_inference() == inference
            assert np.array_equal(call(wz), zero)
            wz.fill_(3)
            assert np.array_equal(call(wz), other)
            wz.zero_()
            assert np.array_equal(call(wz), zero)
    # an ordinary tensor changed under inference mode
    wz = torch.zeros(16, dtype=torch.int8, device=dev)
    assert np.array_equal(call(wz), zero)
    with torch.inference_mode():
        wz.fill_(3)
        assert np.array_equal(call(wz), other)


def test_weight_zero_points_at_a_reused_address(ops, orc, dev):
    """What was learned about a tensor is not believed of the next one at its address."""
    call, want = _conv_case(ops, orc, dev)
    zero, other = want(np.zeros(16, np.int8)), want(np.full(16, 3, np.int8))
    addresses = []
    for value, expect in ((0, zero), (3, other), (0, zero)):
        wz = torch.full((16,), value, dtype=torch.int8, device=dev)
        addresses.append(wz.data_ptr())
        assert np.array_equal(call(wz), expect)
        del wz
    assert len(set(addresses)) < 3  # the allocator did hand the block out again


def test_error_inside_a_call_is_raised(ops, dev):
    """A tensor without storage (here: a batched one) throws when the body asks for its address, at a point where the interpreter lock is given up."""
    x = torch.rand((4, 8), device=dev)
    for _ in range(2):
        with pytest.raises(RuntimeError):
            torch.vmap(lambda t: ops.QuantizeLinear(t, 0.1))(x)
    assert ops.QuantizeLinear(x, 1.0).shape == x.shape


def test_scratch_of_two_streams(ops, orc, dev):
    """Calls that fill scratch (repacked operands, column terms, NHWC copies, packed weights, stem blocks), overlapping on two streams with operands of
    their own: the results of the calls one after the other."""
    gen = torch.Generator(device=dev).manual_seed(7)
    u8 = lambda *s: torch.randint(0, 256, s, dtype=torch.uint8, device=dev, generator=gen)  # noqa: E731
    s8 = lambda *s: torch.randint(-127, 128, s, dtype=torch.int8, device=dev, generator=gen)  # noqa: E731
    z = torch.tensor([9], dtype=torch.uint8, device=dev)

    def problem():
        a, b, x, w, xs, wst = u8(256, 2048), s8(2048, 2048), u8(4, 128, 28, 28), s8(128, 128, 3, 3), u8(8, 3, 112, 112), s8(64, 3, 7, 7)
        ws, wz = torch.rand(128, device=dev, generator=gen) * 1e-3 + 1e-3, torch.full((128,), 3, dtype=torch.int8, device=dev)
        pk = ops.PackedConv(wst, wz[:64] * 0, xs.shape, (2, 2), (3, 3), x_layout=ops.NCHW)
        return [lambda: ops.MatMulInteger(a, b, z, None),
                lambda: ops.QLinearMatMul(a, 0.01, np.uint8(9), b, 0.01, np.int8(0), 30.0, np.uint8(9)),
                lambda: ops.ConvInteger(x, w, np.uint8(9), None, (1, 1), (1, 1)),
                lambda: ops.QLinearConv(x, 0.02, np.uint8(9), w, ws, wz, 0.5, np.uint8(99), strides=(1, 1), pads=(1, 1)),
                lambda: ops.ConvIntegerPacked(xs, pk, np.uint8(3))]

    problems = [problem(), problem()]
    want = [[f() for f in p] for p in problems]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(8):
        for i in range(len(problems[0])):
            for k in range(2):
                with torch.cuda.stream(streams[k]):
                    got[k].append((i, problems[k][i]()))
    torch.cuda.synchronize()
    for k in range(2):
        for i, y in got[k]:
            assert torch.equal(y, want[k][i]), (k, i)
    ops.device_status()


def test_other_threads_run_while_a_zero_point_is_read(ops, orc, dev):
    """A weight zero point that the body has not seen is read from the device, behind whatever the stream has queued: that wait must not keep other
    Python threads from running."""
    call, want = _conv_case(ops, orc, dev)
    expect = want(np.zeros(16, np.int8))
    fresh = [torch.zeros(16, dtype=torch.int8, device=dev) for _ in range(2)]
    call(fresh[0])  # everything loaded
    done = []

    def body():
        torch.cuda._sleep(1_000_000_000)  # about half a second of this thread's stream
        done.append(call(fresh[1]))

    thread = threading.Thread(target=body)
    worst, last = 0.0, time.perf_counter()
    thread.start()
    while thread.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        worst, last = max(worst, now - last), now
    thread.join()
    assert np.array_equal(done[0], expect)
    assert worst < 0.2, "the main thread stood still for %.2f s" % worst
