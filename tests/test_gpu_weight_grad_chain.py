"""How exact the tcgen05 weight gradient is, by the length of its accumulators' chains.

A tensor-memory accumulator is rounded towards zero at each MMA that adds to it.  With positive operands
that loses half a unit in the last place of the running sum an MMA on average, at most 2^-24 of the final
sum: a block that takes `levels` levels of tiles (eight MMAs of 16 points a level and accumulator) loses up
to 8 levels 2^-24.  The level chunks are picked so that a block takes these many levels on 152 SMs, and
longer chains, though quicker by a few steps, are less exact."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,levels", [((128, 128, 64), 56), ((96, 80, 60), 24), ((128, 96, 40), 26)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
@pytest.mark.parametrize("cin,cout,gstride", [(32, 32, 32), (16, 32, 32)])
def test_chain_of_accumulations(built_lib, dims, levels, cin, cout, gstride):
    torch = pytest.importorskip("torch")
    from lex_gb300 import _lib, sgs_cnn
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the chunks follow the number of SMs")
    nx, ny, nz = dims
    n = nx * ny * nz
    gen = torch.Generator(device="cpu").manual_seed(1)
    x = torch.rand(n, cin, generator=gen).cuda().bfloat16()
    g = torch.zeros(n, gstride, device="cuda", dtype=torch.bfloat16)
    g[:, :cout] = torch.rand(n, cout, generator=gen).cuda().bfloat16()
    dw = torch.zeros(27, cout, cin, device="cuda")
    _lib.check(built_lib.lexgb_cnn_conv3d_dw(nx, ny, nz, cin, cout, gstride, sgs_cnn._p(x), sgs_cnn._p(g),
                                             sgs_cnn._p(dw), None, sgs_cnn._stream()))
    xp = torch.nn.functional.pad(x.double().reshape(nz, ny, nx, cin), (0, 0, 1, 1, 1, 1, 1, 1))
    gd = g[:, :cout].double()
    ref = torch.stack([gd.t() @ xp[o // 9:o // 9 + nz, o // 3 % 3:o // 3 % 3 + ny, o % 3:o % 3 + nx].reshape(n, cin)
                       for o in range(27)])
    err = float((dw.double() - ref).norm() / ref.norm())
    assert err <= 8 * levels * 2.0 ** -24, err
