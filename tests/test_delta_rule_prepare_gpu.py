"""q, k, v, step sizes and decays of the gated delta rule: a prompt's tokens eight at a time (gdr_prepare_run_kernel) give the bits of the same
tokens one by one (gdr_prepare_kernel, which also moves the convolution's state on), whatever the portions' lengths and places."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, TAPS = "cuda", 4


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("G,D,H,Dv", [(1, 32, 1, 32), (2, 128, 4, 128), (3, 96, 3, 64)])
@pytest.mark.parametrize("lengths", [[1, 1], [2, 7, 1, 3], [8], [9, 8, 15], [40, 1]], ids=str)
def test_runs_give_the_bits_of_single_tokens(lengths, G, D, H, Dv, dtype):
    from imp_b200 import capi
    lib = capi.load()
    g = torch.Generator().manual_seed(sum(lengths) * D)
    T, n, C = sum(lengths), len(lengths), 2 * G * D + H * Dv
    ld = (C + H * Dv + 2 * H + 7) // 8 * 8
    proj = torch.randn(T, ld, generator=g).to(DEV, dtype)
    w, a_log, dt = torch.randn(C, TAPS, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    first_state = torch.randn(n + 1, TAPS - 1, C, generator=g).to(DEV)
    slots = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    sizes = (G * D, G * D, H * Dv, H, H)

    def call(rows, state, seq, starts, slot, form):        # form: tokens a warp
        update = int(form == 1)
        out = [torch.full((len(rows), m), float("nan"), device=DEV) for m in sizes]
        seq, starts = torch.tensor(seq, dtype=torch.int32, device=DEV), torch.tensor(starts, dtype=torch.int32, device=DEV)
        rc = lib.imp_gdr_prepare_form(ptr(rows), ctypes.c_int64(ld), ptr(w), TAPS, ptr(state), ptr(seq), ptr(starts), ptr(slot), len(rows), len(starts) - 1, G, D, H, Dv,
                                 ptr(a_log), ptr(dt), *map(ptr, out), update, 0 if dtype == torch.float32 else 1, ptr(status), form, stream)
        assert rc == 0
        torch.cuda.synchronize()
        return out

    at = [sum(lengths[:i]) for i in range(n + 1)]
    state = first_state.clone()
    whole = call(proj, state, [i for i, m in enumerate(lengths) for _ in range(m)], at, slots, 8)
    assert torch.equal(state, first_state)
    for i in range(n):
        for t in range(at[i], at[i + 1]):
            one = call(proj[t:t + 1].contiguous(), state, [0], [0, 1], slots[i:i + 1].contiguous(), 1)
            for a, b in zip(whole, one):
                assert torch.equal(a[t], b[0]), (i, t)
    assert int(status) == 0
