"""A kept step in a graph of the caller's: lexgb_step_keep only launches and copies, so a caller may capture
the bound stream around it, however often the pass ran before (from its third run on it is a graph itself)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [0, 1, 4])
def test_kept_step_can_be_captured(built_lib, before):
    import torch
    from lex_gb300 import _lib, autograd as lag
    from test_gpu_substep_chain import solver, state
    dims = (20, 12, 10)
    S, qv0 = solver(*dims)
    side = torch.cuda.Stream()
    with S, torch.cuda.stream(side):
        x = state(*dims, qv0)
        keep = lambda: _lib.check(S.lib.lexgb_step_keep(S.handle))
        g = [torch.randn(t.shape, generator=torch.Generator(device="cpu").manual_seed(5)).cuda() for t in x]

        def reverse():
            out = [torch.empty_like(t) for t in x]
            _lib.check(S.lib.lexgb_step_vjp_kept(S.handle, lag._ptrs(g), lag._ptrs(out), 1))
            return out
        lag.set_state(S, x, raw=True)
        keep()
        ref = list(lag.get_state(S, raw=True)) + reverse()
        for _ in range(before):
            lag.set_state(S, x, raw=True)
            keep()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin(capture_error_mode="thread_local")
        keep()
        graph.capture_end()
        for _ in range(2):
            lag.set_state(S, x, raw=True)
            graph.replay()
            got = list(lag.get_state(S, raw=True)) + reverse()
            torch.cuda.synchronize()
            for i, (a, b) in enumerate(zip(got, ref)):
                assert torch.equal(a, b), i
