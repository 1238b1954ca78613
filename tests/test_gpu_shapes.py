"""Sizes where the kernels' splits change: blocks of the allocation-free matmul, the operand ring's cuts and the tile plan's edges,
attention over one and two accumulator halves, results that leave through the pinned ring."""
import numpy as np
import pytest

import harness
from aspen_b200 import api, cfgs, weights
from oracle import port
from test_zz_no_alloc import oracle_matmul

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,m", [(1, 1, 1), (2, 130, 33), (4, 128, 9), (8, 257, 64), (9, 31, 32), (33, 1021, 31), (65, 64, 129), (190, 66, 700), (700, 40, 641)])
@pytest.mark.parametrize("act", [0, 4, 8])
def test_noalloc_blocks_at_their_edges(n, k, m, act):
    import torch
    rng = np.random.default_rng(n * 1000 + k)
    x = rng.standard_normal((n, k), dtype=np.float32)
    w = (rng.standard_normal((m, k), dtype=np.float32) / np.sqrt(k)).astype(np.float32)
    b = rng.standard_normal((m,), dtype=np.float32)
    xd, wd, bd = (torch.from_numpy(a).cuda() for a in (x, w, b))
    od = torch.full((n, m), float("nan"), device="cuda")
    torch.cuda.synchronize()
    rc = api.lib().aspen_b200_matmul_noalloc(xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), od.data_ptr(), n, k, m, act, None)
    assert rc == 0, api.last_error()
    want = oracle_matmul(x, w, b, act)
    bad, ea, er = harness.compare(od.cpu().numpy(), want, 1e-4, 1e-5 * float(np.abs(want).max()))
    assert bad == 0, f"{bad} mismatches, max abs {ea:.3e}, max rel {er:.3e}"


# Blocks of 128 columns x 64 or 128 rows and chunks of 32 of k, at their edges, with every kind of load (k % 4, k % 2, odd), one block an SM
# and several, and the kernel that runs them (test_native.py).
SPLIT_SHAPES = [(4100, 256, 2050, "split 128"), (4100, 319, 2050, "split 128"), (1283, 518, 1304, "split 128"), (1283, 516, 1301, "split 128"),
                (385, 1000, 2047, "split 64"), (385, 1002, 2048, "split 64"), (377, 1001, 2049, "split 64")]
RANGE_SHAPES = [(1283, 514, 1301, "split 128"), (385, 1000, 2047, "split 64")]


def noalloc(x, w, b, act):
    import torch
    xd, wd, bd = (None if a is None else torch.from_numpy(a).cuda() for a in (x, w, b))
    od = torch.full((x.shape[0], w.shape[0]), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert api.lib().aspen_b200_matmul_noalloc(xd.data_ptr(), wd.data_ptr(), None if b is None else bd.data_ptr(), od.data_ptr(), x.shape[0], x.shape[1], w.shape[0], act, None) == 0, api.last_error()
    return od.cpu().numpy()


@pytest.mark.parametrize("n,k,m,kernel", SPLIT_SHAPES)
@pytest.mark.parametrize("act,with_bias", [(0, False), (0, True), (3, True), (8, True)])
def test_noalloc_on_the_tensor_cores_is_as_close_to_64_bits_as_fp32_sums(n, k, m, kernel, act, with_bias):
    """A sum of k products rounded to fp32 one after the other is off by some 0.2 sqrt(k / 2) 2**-24 of its size where two sums are kept (the FMA
    blocks); 2**-23 covers the rounding of the result and of the activation on top."""
    rng = np.random.default_rng(n + k)
    x = rng.standard_normal((n, k), dtype=np.float32)
    w = (rng.standard_normal((m, k)) * np.sqrt(2 / k)).astype(np.float32)
    b = rng.standard_normal((m,), dtype=np.float32) if with_bias else None
    got = noalloc(x, w, b, act)
    want = x.astype(np.float64) @ w.T.astype(np.float64) + (b if with_bias else 0)
    if act == 3:
        want = np.tanh(want)
    elif act == 8:
        import torch
        want = torch.nn.functional.gelu(torch.from_numpy(want)).numpy()
    assert np.isfinite(got).all()
    assert np.linalg.norm(got - want) <= (0.2 * np.sqrt(k / 2) * 2.0**-24 + 2.0**-23) * np.linalg.norm(want)


@pytest.mark.parametrize("n,k,m,kernel", [(1283, 3072, 1301, "split 128"), (385, 3072, 2048, "split 64")])
def test_noalloc_on_the_tensor_cores_adds_chunks_two_by_two(n, k, m, kernel):
    """Operands of one sign, whose partial sums grow evenly: k / 64 additions to a total, each off by 0.42 2**-24 of it in the root mean square (see
    below), come to 0.42 sqrt(k / 64 / 3), and the accumulators of a chunk cut off up to a unit twice, at half the sum and at all of it, 1.1 2**-24
    together.  (With every chunk added to the total by itself it is 2.4 2**-24, past this bound.)"""
    rng = np.random.default_rng(k + m)
    x, w = np.abs(rng.standard_normal((n, k), dtype=np.float32)), np.abs(rng.standard_normal((m, k), dtype=np.float32))
    got, want = noalloc(x, w, None, 0), x.astype(np.float64) @ w.T.astype(np.float64)
    assert np.linalg.norm(got - want) <= np.sqrt(0.42**2 * k / 192 + 1.1**2) * 2.0**-24 * np.linalg.norm(want)


@pytest.mark.parametrize("n,k,m,kernel", [(1283, 3072, 1301, "split 128"), (385, 3070, 2047, "split 64")])
def test_noalloc_blocks_with_infinities_cost_what_fp32_blocks_do(n, k, m, kernel):
    """One value of each block is an infinity: the SM that had it computes it again in 32 x 32 fp32 blocks, one after another, which takes
    four times as long as the tensor cores (value by value 43 and 95 times).  Rounding to nearest is off by 0.42 2**-24 of
    a value in the root mean square (0.58 2**-24 over the mantissa); two sums of k / 2 products, whose partial sums grow with the square root, end up
    off by 0.42 sqrt(k) / 2 = 0.3 sqrt(k / 2) units."""
    import time
    rng = np.random.default_rng(k)
    x = rng.standard_normal((n, k), dtype=np.float32)
    w = (rng.standard_normal((m, k)) * np.sqrt(2 / k)).astype(np.float32)

    def best():
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            rc = api.lib().aspen_b200_matmul_noalloc(xd.data_ptr(), wd.data_ptr(), None, od.data_ptr(), n, k, m, 0, None)
            t.append(time.perf_counter() - t0)
            assert rc == 0, api.last_error()
        return min(t)

    import torch
    xd, wd, od = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), torch.full((n, m), float("nan"), device="cuda")
    torch.cuda.synchronize()
    finite = best()
    rows, cols = np.arange(7, m, 64), np.arange(5, n, 128)
    w[rows, 3] = np.inf
    x[cols, 2] = -np.inf
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    assert best() < 10 * finite
    got = od.cpu().numpy()
    with np.errstate(all="ignore"):
        want = x.astype(np.float64) @ w.T.astype(np.float64)
    plain = np.ix_(~np.isin(np.arange(n), cols), ~np.isin(np.arange(m), rows))
    assert np.isfinite(got[plain]).all() and np.linalg.norm(got[plain] - want[plain]) <= (0.3 * np.sqrt(k / 2) * 2.0**-24 + 2.0**-23) * np.linalg.norm(want[plain])
    other = np.ones((n, m), bool)
    other[plain] = False
    np.testing.assert_array_equal(got[other], want[other].astype(np.float32))


@pytest.mark.parametrize("n,k,m,kernel", RANGE_SHAPES)
def test_noalloc_on_the_tensor_cores_over_the_range_of_fp32(n, k, m, kernel):
    """Infinities and NaN spread as in a sum of fp32 products, and only into their own rows and columns; large, small and denormal values keep
    the precision of fp32 products, those whose last bits no bf16 part holds (below 2**-110) and those whose products are denormal included."""
    rng = np.random.default_rng(3)
    x = rng.standard_normal((n, k), dtype=np.float32)
    w = (rng.standard_normal((m, k)) * np.sqrt(2 / k)).astype(np.float32)
    w[w == 0] = 1
    scaled = {10: -100, 11: -109, 12: -112, 13: -116, 14: -120, 15: -126, 16: -132, 17: 60, 150: -100, 151: -105, 152: -60, 153: -70, 154: -75, 280: -120, 281: 60}
    for row, e in scaled.items():
        x[row] *= np.float32(2.0**e)
    x[18] = rng.uniform(1, 2, k).astype(np.float32) * np.float32(2.0**-127)
    x[19] = np.exp(-rng.uniform(0, 103, k)).astype(np.float32)           # probabilities, down to denormal ones
    x[282, ::2] = 0
    parts = {"large": slice(20, 120), "small": slice(120, 220), "smaller": slice(220, 320), "plain": slice(320, m)}
    w[parts["large"]] *= np.float32(2.0**60)
    w[parts["small"]] *= np.float32(2.0**-60)
    w[parts["smaller"]] *= np.float32(2.0**-122)
    x[3, 7], x[300, 100], x[n - 1, k - 1], x[301, 5] = np.inf, -np.inf, np.nan, np.float32(3.4e38)
    w[320:, 5] = np.float32(1e-3)
    w[parts["large"], 5] = np.float32(1e-3)          # 3.4e38 times a value of 2**60 would be past the range of fp32
    got = noalloc(x, w, None, 0)
    with np.errstate(all="ignore"):
        want = x.astype(np.float64) @ w.T.astype(np.float64)
    special = np.isin(np.arange(n), (3, 300, n - 1))
    np.testing.assert_array_equal(got[[3, 300]], want[[3, 300]].astype(np.float32))        # every sum is an infinity of w's sign
    assert np.isnan(got[n - 1]).all() and np.isfinite(got[~special]).all()
    scale = np.abs(x[~special].astype(np.float64)) @ np.abs(w.T.astype(np.float64))        # each product is off by 2**-24 at most, each of some k partial sums too
    assert (np.abs(got[~special] - want[~special]) <= 2.0**-24 * (1 + np.sqrt(k)) * scale + 2.0**-149 * k).all()
    # two sums of k / 2 products in the root mean square (see above; over 100 outputs that scatters by 7 %, so 2**-23 on top leaves four times
    # that), and half a unit of 2**-149 an addition where they are denormal
    for row in (*scaled, 18, 19, 282):
        for name, cols in parts.items():
            off, size = (np.linalg.norm(v) for v in (got[row, cols] - want[row, cols], want[row, cols]))
            assert off <= (0.3 * np.sqrt(k / 2) * 2.0**-24 + 2.0**-23) * size + 2.0**-150 * np.sqrt(k * (cols.stop - cols.start)), (row, name, off / size)


@pytest.mark.parametrize("n,k,m,kernel", RANGE_SHAPES)
@pytest.mark.parametrize("act", [0, 4])          # 4: ReLU, which makes a zero of a NaN
def test_noalloc_on_the_tensor_cores_where_finite_operands_overflow(n, k, m, kernel, act):
    """Sums past the range of fp32 are infinities, also where the products of the operands' parts overflow with either sign; sums within it are
    right although a product of rounded parts is past it.  Row 5 of x and row 9 of w lie in one block, rows 130 and 300 in others."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, k), dtype=np.float32)
    w = (rng.standard_normal((m, k)) * np.sqrt(2 / k)).astype(np.float32)
    x[5] = np.float32(1.1e25) * (1 + rng.random(k, dtype=np.float32) / 64)
    w[9] = np.float32(1.3e25) * (1 + rng.random(k, dtype=np.float32) / 64)          # 1.4e50 a product
    w[10] = -w[9]
    x[130], w[200] = 0, 0
    x[130, 3], w[200, 3] = np.float32(1.9975), np.float32(2.0**127)          # within the range; 2 * 2**127, as the first part rounds, is not
    x[300], w[201] = 0, 0
    x[300, ::2] = w[201, ::2] = np.float32(1.8e19)                                    # each product within the range, their sum past it
    got = noalloc(x, w, None, act)
    with np.errstate(over="ignore"):
        want = (x.astype(np.float64) @ w.T.astype(np.float64)).astype(np.float32)
    if act == 4:
        want = np.maximum(want, 0)
    far = np.isinf(want)
    assert far[5, 9] and far[300, 201] and (far[5, 10] or act == 4) and np.isfinite(want[130, 200]) and want[130, 200] > np.float32(3.3e38)
    np.testing.assert_array_equal(got[far], want[far])
    assert np.isfinite(got[~far]).all()
    scale = np.abs(x.astype(np.float64)) @ np.abs(w.T.astype(np.float64))        # as above
    assert (np.abs(got[~far].astype(np.float64) - want[~far]) <= (2.0**-24 * (1 + np.sqrt(k)) * scale + 2.0**-149 * k)[~far]).all()


@pytest.mark.parametrize("name,batch,seq,precision", [("tiny_attn", 1, 1, 0), ("tiny_attn", 3, 33, 0), ("tiny_attn", 1, 129, 0), ("tiny_attn_causal", 2, 255, 0),
                                                      ("tiny_attn_causal", 1, 257, 0), ("tiny_attn_causal", 1, 300, 1), ("tiny_transformer", 64, 128, 0),
                                                      ("tiny_cnn", 1, 0, 0), ("tiny_cnn", 33, 0, 0), ("tiny_cnn", 9, 0, 1), ("custom", 1, 0, 0), ("custom", 130, 0, 0),
                                                      ("custom", 3, 0, 1), ("custom", 2, 0, 0), ("custom", 5, 0, 0), ("custom", 8, 0, 0), ("custom", 9, 0, 0),
                                                      ("custom", 8, 0, 1), ("tiny_attn", 1, 7, 1),
                                                      ("tiny_heads80", 2, 40, 0), ("tiny_heads80", 1, 300, 0), ("tiny_heads80", 1, 40, 1), ("tiny_heads12", 3, 130, 0),
                                                      ("tiny_gpt", 1, 512, 0), ("tiny_attn", 1, 520, 0), ("tiny_attn_causal", 1, 520, 1), ("tiny_transformer", 1, 5, 0), ("tiny_cnn", 4, 0, 0)])
def test_every_layer_at_the_edges_of_the_plan(name, batch, seq, precision, workdir):
    every_layer_matches(name, batch, seq, precision, 1, workdir)


@pytest.mark.parametrize("name,batch,seq", [("tiny_heads10", 2, 40), ("tiny_heads12", 3, 24), ("tiny_heads10", 1, 9), ("tiny_cnn", 2, 0), ("tiny_acts", 3, 0)])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("plan,quanta", [("1", None), ("0", None), ("0", (10, 12)), ("0", (6, 40))])
def test_tiles_that_start_anywhere(name, batch, seq, precision, plan, quanta, workdir, monkeypatch):
    """Heads of ten or twelve features, and graphs executed with their own tiles (ASPEN_B200_PLAN=0) of odd heights: rows and strides that
    are no multiple of four, in every kind of tile."""
    monkeypatch.setenv("ASPEN_B200_PLAN", plan)
    if quanta:
        api.lib().aspen_b200_set_tile_quanta(*quanta, 100000)
    every_layer_matches(name, batch, seq, precision, 2 if quanta else 0, workdir)


def every_layer_matches(name, batch, seq, precision, profile, workdir):
    cfg, wf = harness.prepare(name, workdir)
    dev = harness.Device(cfg, wf, batch, seq, 20, precision, profile)
    x = harness.make_input(name, dev.input_shape())
    for _ in range(2):                                        # a second pass over the same memory
        assert dev.run(x) == 0, api.last_error()
    kw, scheme, (wseed, _) = harness.NETS[name]
    text, wl = cfgs.BUILDERS[harness._BUILDER.get(name, name)](**kw)
    outs = port.run(text, weights.make_weights(wl, wseed, scheme), x, batch, seq)
    layers_match(dev, outs, precision)
    dev.close()


def layers_match(dev, outs, precision):
    for i in range(1, dev.nasm.num_ldata):
        got, want = dev.nasm.ldata(i), outs[i]
        scale = float(np.abs(want).max())
        if precision == 1:
            bad, ea, er = harness.compare(got, want, 1e-4, 1e-5 * scale)
            assert bad == 0, f"layer {i}: {bad} mismatches, max abs {ea:.3e}, max rel {er:.3e}"
        else:
            assert float(np.abs(got.astype(np.float64) - want).max()) <= 1e-2 * scale, f"layer {i}"


def _conv_net(side, channels, layers, out):
    """cfg and weighted layers: convolutions (channels, size, stride, pad) one after the other and a connected layer over the last."""
    text, wl = f"[net]\nheight={side}\nwidth={side}\nchannels={channels}\n\n", []
    for c, size, stride, pad in layers:
        text += f"[convolutional]\nfilters={c}\nsize={size}\nstride={stride}\npad={pad}\nactivation=relu\n\n"
        wl.append(("conv", (c, channels, size, size), channels * size * size))
        side, channels = (side + 2 * pad - size) // stride + 1, c
    wl.append(("fc", (out, channels, side, side), channels * side * side))
    return text + f"[connected]\noutput={out}\nactivation=linear\n", wl


def test_launches_of_more_sets_of_graphs_than_are_kept(workdir):
    """92 sets of seven graphs in turn, without a stop between them: the order of one is written where another's was."""
    import itertools
    dnn = api.Dnn(*harness.prepare("custom", workdir))
    graphs = [api.Nasm(dnn, b, 0, 8) for b in (1, 2, 3, 5, 8, 13, 21)]
    rpool, group = api.Rpool(), api.DseGroup(0, 0)
    group.set_rpool(rpool)
    xs = [harness.make_input("custom", (g.ldata_info(0)["W"], g.ldata_info(0)["H"])) for g in graphs]
    first = {}
    for _ in range(2):
        for owed in itertools.chain(*(itertools.combinations(range(7), r) for r in (7, 2, 3, 4))):
            for i in owed:
                rpool.add(graphs[i], xs[i])
            group.run()
            for i in owed:
                group.wait(graphs[i])
            assert group.status() == 0, api.last_error()
            for i in owed:
                got = graphs[i].ldata(graphs[i].num_ldata - 1).copy()
                np.testing.assert_array_equal(got, first.setdefault(i, got))
    group.stop()
    assert len(first) == 7 and all(np.abs(v).max() > 0 for v in first.values())
    group.close()
    for o in (*graphs, rpool, dnn):
        o.close()


@pytest.mark.parametrize("batch,side,channels,layers", [
    (3, 30, 3, [(48, 7, 2, 3), (24, 3, 1, 1), (33, 3, 2, 1), (64, 1, 2, 0), (10, 1, 1, 0)]),       # rows of 15 pixels; channels no multiple of 32, or of 4
    (12, 37, 1, [(20, 11, 4, 2), (96, 3, 1, 0), (12, 5, 1, 2)]),                                   # one channel, a window of two chunks a row
    (9, 18, 4, [(40, 3, 1, 1), (6, 3, 3, 2), (70, 2, 1, 1)]),
    (11, 9, 3, []),                                                                                # connected straight to the image
    (2, 17, 9, [(5, 3, 1, 1), (36, 4, 2, 1)]),                                                     # an input of more than four channels
    (2, 21, 3, [(36, 3, 1, 4), (40, 3, 9, 1)])])                                                   # windows that lie in the padding, a stride past TMA's: fp32 blocks
@pytest.mark.parametrize("precision", [0, 1])
def test_convolutions_of_any_channel_count_and_width(batch, side, channels, layers, precision, workdir):
    text, wl = _conv_net(side, channels, layers, 13)
    cfg, wf = f"{workdir}/conv_{side}.cfg", f"{workdir}/conv_{side}.bin"
    with open(cfg, "w") as f:
        f.write(text)
    ws = weights.make_weights(wl, 41, "he")
    weights.write_aspen_data(wf, ws)
    dev = harness.Device(cfg, wf, batch, 0, 20, precision, 1)
    x = np.random.default_rng(side).standard_normal(dev.input_shape(), dtype=np.float32)
    for _ in range(2):
        assert dev.run(x) == 0, api.last_error()
    layers_match(dev, port.run(text, ws, x, batch, 0), precision)
    dev.close()


@pytest.mark.parametrize("batch,seq", [(1, 7), (2, 45), (1, 130)])
@pytest.mark.parametrize("precision", [0, 1])
def test_attention_over_values_of_any_layer(batch, seq, precision, workdir):
    """Values without a projection of their own: a layernorm's output (twice), the network's input, a residual add, and a residual add
    that would otherwise be computed by its producer."""
    d, h = 64, 2
    k, v = f"n_head={h}\nn_embd={d}\n", f"[attention_v]\nM={d}\nn_head={h}\nn_embd={d}\n"
    text = (f"[net]\nM={d}\nheight=1\nfilters={d}\n\n[layernorm]\nM={d}\n\n[matmul]\nM={d}\n{k}\n[matmul]\nM={d}\nparent=-2\n{k}\n"
            f"[attention_k]\nparent=-1\nfrom=-2\nM=1\nK={d // h}\n{k}\n{v}parent=-1\nfrom=-4\n\n{v}parent=-2\nfrom=-5\n\n{v}parent=-3\nfrom=-7\n\n"
            f"[shortcut]\nfrom=-3\nM={d}\n\n{v}parent=-5\nfrom=-1\n\n[matmul]\nM={d}\n\n[shortcut]\nfrom=-2\nM={d}\n\n{v}parent=-8\nfrom=-1\n\n")
    cfg, wf = f"{workdir}/values.cfg", f"{workdir}/values.bin"
    with open(cfg, "w") as f:
        f.write(text)
    ws = weights.make_weights([("layernorm", (d,), d)] + [("matmul", (d, d), d)] * 3, 43, "he")
    weights.write_aspen_data(wf, ws)
    dev = harness.Device(cfg, wf, batch, seq, 20, precision, 1)
    x = np.random.default_rng(seq).standard_normal(dev.input_shape(), dtype=np.float32)
    for _ in range(2):
        assert dev.run(x) == 0, api.last_error()
    layers_match(dev, port.run(text, ws, x, batch, seq), precision)
    dev.close()


@pytest.mark.parametrize("channels", [200704, 300000])
def test_connected_layer_over_more_channels_than_a_product_of_indices_can_hold(channels, workdir):
    """fp32 blocks find the channel of a k by a multiplication; k times the channel count passes 2^32 here.  The last pieces of k
    carry most of the sum, so one that is taken as lying outside the image shows."""
    n, m = 9, 16
    rng = np.random.default_rng(channels)
    x = rng.standard_normal((n, channels), dtype=np.float32)
    x[:, -64:] *= 100.0
    w = (rng.standard_normal((m, channels), dtype=np.float32) / np.sqrt(channels)).astype(np.float32)
    b = rng.standard_normal((m,), dtype=np.float32)
    cfg, wf = f"{workdir}/wide_{channels}.cfg", f"{workdir}/wide_{channels}.bin"
    with open(cfg, "w") as f:
        f.write(f"[net]\nheight=1\nwidth=1\nchannels={channels}\n\n[connected]\noutput={m}\nactivation=linear\n")
    weights.write_aspen_data(wf, [(w.reshape(m, channels, 1, 1), b)])
    dev = harness.Device(cfg, wf, n, 0, 4, precision=1, profile=1)
    assert dev.run(x) == 0, api.last_error()
    want = x.astype(np.float64) @ w.astype(np.float64).T + b
    bad, ea, er = harness.compare(dev.nasm.ldata(1), want, 1e-4, 1e-5 * float(np.abs(want).max()))
    dev.close()
    assert bad == 0, f"{bad} mismatches, max abs {ea:.3e}, max rel {er:.3e}"


_ACT64 = {"logistic": lambda x: 1.0 / (1.0 + np.exp(-x)), "tanh": np.tanh, "leaky": lambda x: np.where(x > 0, x, 0.1 * x),
          "elu": lambda x: np.where(x > 0, x, 0.1 * (np.exp(x) - 1.0)), "selu": lambda x: np.where(x > 0, 1.0507 * x, 1.0507 * 1.67326 * (np.exp(x) - 1.0))}


@pytest.mark.parametrize("act", sorted(_ACT64))
def test_activations_of_the_tensor_core_epilogue_are_rounded_once(act, workdir):
    """Matmul and fused residual add, outputs from 1e-7 to 10: the activation of what the same network gives with `linear`, in 64 bits,
    to the last place of fp32 (the reference's double-precision forms, src/naive_kernels.c:11-57)."""
    d, n = 96, 70
    rng = np.random.default_rng(31)
    x = (rng.standard_normal((n, d)) * 10.0 ** rng.uniform(-7, 1, (n, 1))).astype(np.float32)
    ws = [((rng.standard_normal((d, d)) / np.sqrt(d)).astype(np.float32), np.zeros(d, np.float32)) for _ in range(2)]
    wf = f"{workdir}/act_{act}.bin"
    weights.write_aspen_data(wf, ws)
    outs = []
    for a in ("linear", act):
        cfg = f"{workdir}/act_{act}_{a}.cfg"
        with open(cfg, "w") as f:
            f.write(f"[net]\nM={d}\nheight=1\nfilters={d}\n\n[matmul]\nM={d}\nactivation={a}\n\n[matmul]\nM={d}\nparent=-2\n\n"
                    f"[shortcut]\nfrom=-3\nM={d}\nactivation={a}\n\n")
        dev = harness.Device(cfg, wf, 1, n, 4, 0, 1)
        assert dev.run(x) == 0, api.last_error()
        outs.append([dev.nasm.ldata(i).copy() for i in (1, 3)])
        dev.close()
    for layer, lin, got in zip((1, 3), *outs):
        want = _ACT64[act](lin.astype(np.float64))
        assert float(np.abs(want).max()) > 0
        off = np.abs(got.astype(np.float64) - want) / np.spacing(np.abs(want).astype(np.float32))
        assert float(off.max()) <= 1.0, f"layer {layer}: {off.max():.1f} units in the last place at {lin.ravel()[off.argmax()]:.3e}"


@pytest.mark.parametrize("precision", [0, 1])
def test_launches_of_changing_sets_of_graphs(precision, workdir):
    """A launch's tiles are handed out in an order made for the graphs that owe a pass: one alone, several together, another several."""
    names = ("tiny_cnn", "tiny_transformer", "custom")
    dnns = [api.Dnn(*harness.prepare(n, workdir)) for n in names]
    graphs = [api.Nasm(d, 2, 16 if n == "tiny_transformer" else 0, 8) for d, n in zip(dnns, names)]
    rpool, group = api.Rpool(), api.DseGroup(0, precision)
    group.set_rpool(rpool)
    xs = [harness.make_input(n, (g.ldata_info(0)["W"], g.ldata_info(0)["H"])) for n, g in zip(names, graphs)]
    alone = {}
    for owed in ((0,), (1,), (2,), (0, 1, 2), (1, 2), (0, 2), (1, 2), (0,)):
        for i in owed:
            rpool.add(graphs[i], xs[i])
        group.run()
        for i in owed:
            group.wait(graphs[i])
        group.stop()
        assert group.status() == 0, api.last_error()
        for i in owed:
            got = graphs[i].ldata(graphs[i].num_ldata - 1).copy()
            np.testing.assert_array_equal(got, alone.setdefault(i, got))
    assert len(alone) == 3 and all(np.abs(v).max() > 0 for v in alone.values())
    group.close()
    for o in (*graphs, rpool, *dnns):
        o.close()


@pytest.mark.parametrize("batch,side,channels,layers", [
    (1, 7, 64, [(50, 3, 1, 1), (30, 3, 1, 1), (514, 1, 1, 0), (33, 3, 2, 1)]),       # k 576, 450, 30, 4626: rows that are no multiple of four
    (3, 5, 66, [(64, 5, 1, 2), (130, 3, 1, 1)]),                                     # k 1650, 576; channels that are no multiple of four
])
@pytest.mark.parametrize("act", ["relu", "logistic"])
def test_fp32_layers_whose_k_is_shared_by_several_tiles(batch, side, channels, layers, act, workdir):
    """Launched alone in the fp32 mode, layers of few tiles split their k; whichever tile comes last adds the sums in the same order, so
    a run's bits are those of the run before."""
    text, wl = _conv_net(side, channels, layers, 20)
    text = text.replace("activation=relu", f"activation={act}")
    cfg, wf = f"{workdir}/share_{channels}_{act}.cfg", f"{workdir}/share_{channels}_{act}.bin"
    with open(cfg, "w") as f:
        f.write(text)
    ws = weights.make_weights(wl, 47, "he")
    weights.write_aspen_data(wf, ws)
    dev = harness.Device(cfg, wf, batch, 0, 20, 1, 1)
    x = np.random.default_rng(side).standard_normal(dev.input_shape(), dtype=np.float32)
    assert dev.run(x) == 0, api.last_error()
    once = [dev.nasm.ldata(i).copy() for i in range(1, dev.nasm.num_ldata)]
    for _ in range(20):
        assert dev.run(x) == 0, api.last_error()
    for i, o in enumerate(once):
        np.testing.assert_array_equal(dev.nasm.ldata(i + 1), o)
    layers_match(dev, port.run(text, ws, x, batch, 0), 1)
    dev.close()
