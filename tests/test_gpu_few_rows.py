"""GEMM launches with fewer rows than a tile, whose loads cover only the rows that exist: row counts around multiples of eight
and the ends of the range, narrow and wide outputs, short and long K, with and without a fused residual Add."""
import numpy as np
import pytest

import graph_cases as G
import opworkloads
import pyb2vx as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [17, 24, 49, 63, 64, 100, 127, 128, 129])
@pytest.mark.parametrize("k,n", [(1040, 48), (336, 320)])
def test_fully_connected(product_lib, oracle_lib, rows, k, n):
    for kind in ("s8pc", "u8"):
        build = G.fc_q(k, n, rows, w_kind=kind)
        want, _ = G.run_case(oracle_lib, build, 11)
        got, kernels = G.run_case(product_lib, build, 11)
        assert any(k["name"].startswith("gemm_i8_tc") for k in kernels)
        G.assert_same(want, got)


@pytest.mark.parametrize("spec,batch", [("convadd:1:64:96:5:1", 1), ("convadd:1:512:64:7:1", 1), ("convadd:1:64:256:7:1", 2), ("convadd:1:96:48:11:1", 1)])
def test_one_tile_with_fused_add(product_lib, oracle_lib, spec, batch):
    outs = []
    for lib in (oracle_lib, product_lib):
        g = B.Graph(lib)
        w = opworkloads.build(spec, batch, g, np.random.default_rng(4))
        g.compile()
        for t, a in w["inputs"]:
            g.write(t, a)
        g.run()
        outs.append([g.read(t) for t in w["outputs"]])
        names = [k["name"] for k in g.kernels()]
        g.close()
    assert any("+add" in n for n in names), names
    G.assert_same(*outs)


@pytest.mark.parametrize("channels", [32, 48, 64, 96, 150, 288])
@pytest.mark.parametrize("form", ["1x1", "3x3", "add"])
def test_one_narrow_tile_for_each_block(product_lib, oracle_lib, launch_rules, channels, form):
    """Launches of about a wave with tiles of 16 to 64 columns: all epilogue warps share the only tile of a block, or, on 19 x 19 at batch
    47 and 75 x 75 at batch 3, where a convolution's spatial tiles are more than a wave and its pixels / 128 are not, teams take them."""
    sizes = ((56, 1), (19, 4), (65, 2), (19, 47), (75, 3), (56, 4))
    ks = [32, 64][form == "add"]
    rules = launch_rules([("conv", b, hw, hw, 3, 1, ks, channels) if form == "3x3" else ("gemm", b * hw * hw, ks, channels) for hw, b in sizes])
    narrow = [one_each for _, _, columns, _, one_each in rules if 32 <= columns <= 64]
    assert 1 in narrow and (form != "3x3" or 0 in narrow), rules
    for hw, batch in sizes:
        if form == "add":
            outs = []
            for lib in (oracle_lib, product_lib):
                g = B.Graph(lib)
                w = opworkloads.build("convadd:1:64:%d:%d:1" % (channels, hw), batch, g, np.random.default_rng(channels))
                g.compile()
                for t, a in w["inputs"]:
                    g.write(t, a)
                g.run()
                outs.append([g.read(t) for t in w["outputs"]])
                g.close()
            G.assert_same(*outs)
        else:
            k = int(form[0])
            build = G.conv2d_q(hw, hw, 32, batch, k, k, channels)
            G.assert_same(*(G.run_case(lib, build, channels)[0] for lib in (oracle_lib, product_lib)))
