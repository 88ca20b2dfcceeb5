"""Bounded waits that ran out on the device, from the host's side (the count is set by hand, no kernel
waits): the call they belong to fails, and the next one on the same context does not."""
import ctypes

import numpy as np
import pytest


def count_waits(wl, ctx, n, unread=False):
    lib = wl.load_library()
    lib.wl_ctx_count_expired_waits.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_int32]
    assert lib.wl_ctx_count_expired_waits(ctx.handle, n, int(unread)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("unread", [False, True])
def test_an_expired_wait_fails_one_call_only(wl, unread):
    log_n = 6
    consts, inputs = wl.generate_workload(log_n)
    with wl.Context(0) as ctx:
        w = wl.Witness.generate(ctx, consts, inputs, log_n)
        table = wl.AirTable(ctx, consts, log_n)
        proof = table.prove_witness(w)

        def verify():
            return list(wl.verify_batch_device(ctx, consts, [(log_n, proof)]))

        assert verify() == [0]
        for call in (lambda: table.prove_witness(w), verify):
            count_waits(wl, ctx, 3, unread)
            if not unread:
                with pytest.raises(wl.ProverError, match="a bounded wait ran out"):
                    call()
            assert np.array_equal(table.prove_witness(w), proof)
            assert verify() == [0]
        w.free()
