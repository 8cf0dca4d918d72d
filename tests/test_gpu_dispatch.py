"""Dispatch rules of the tensor-core convolutions at the sizes where they change: input widths that do not fill the last
64-channel chunk, and batches on either side of the small-batch kernel's limit."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from katago_b200 import capi
from katago_b200 import modelfile as mf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(capi.PRECISION_FP16, 0.03), (capi.PRECISION_BF16, 0.2)])
@pytest.mark.parametrize("trunk,mid", [(16, 24), (32, 48), (96, 96), (112, 40), (80, 200)])
def test_input_widths_between_chunks(prec, tol, trunk, mid, oracle):
    """Residual blocks whose widths end 8 to 56 channels into a 64-channel chunk; the chunk's other channels must count as
    zeros (they lie in the next row of the tensor).  The tolerance is the reference's reduced-precision layer tolerance
    (cpp/tests/testnn.cpp:8-15), widened for bf16's 8 mantissa bits."""
    g = mf._Gen(400 + trunk + mid)
    rng = np.random.default_rng(trunk * mid)
    mask = np.zeros((3, 19, 19), np.float32)
    mask[0] = 1; mask[1, :13, :13] = 1; mask[2, :9, :10] = 1
    layer = mf._gen_ordinary(g, trunk, mid, mf.ACT_MISH)
    x = rng.standard_normal((3, 19, 19, trunk)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, trunk)
    out = capi.eval_layer(blob, x, mask, trunk, precision=prec)
    assert np.all(np.abs(out - ref) <= tol * np.maximum(np.maximum(np.abs(out), np.abs(ref)), 3.0))


def _wide_tiles(test_file, keyword):
    """Runs tests in a process of their own in which no batch is small (the switch is read once per process): their few boards
    then go through the wide-tile kernels and the merged launches."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", os.path.join("tests", test_file), "-k", keyword], cwd=root,
                       env=dict(os.environ, KB_NO_SMALL="1"), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=600)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:]


def test_input_widths_between_chunks_in_wide_tiles():
    _wide_tiles("test_gpu_dispatch.py", "(between_chunks or gpool_widths) and not wide_tiles")


def test_layers_and_nets_in_wide_tiles():
    _wide_tiles("test_gpu_parity.py", "conv_layer_tensor_core or blocks_and_norm_with_masks or nbt_reduced_precision or every_block_at_full_depth")


def test_chains_and_pairs_with_partial_chunks(oracle):
    """Full batches of nets whose widths end inside a 64-channel chunk, a few rows against the oracle: 96 input channels in the
    multi-layer launches, 96 and 160 into 256-wide tiles in CTA pairs.  Tolerance as above."""
    for trunk, mid, n, edge in ((96, 96, 128, 19), (96, 256, 200, 13), (256, 160, 200, 13)):
        blob = mf.to_blob(mf.make_convnet("partial", 460 + mid, 15, trunk, ["plain", "gpool", "plain"], (32, 32, 32, 64), mf.ACT_MISH, mid_c=mid,
                                          regular_c=64, gpool_c=32))
        sizes = ([edge, 9, 7, edge] * n)[:n]
        sp, gl = mf.random_positions(n, seed=14, nn_len=edge, board_sizes=sizes)
        h = capi.Handle(capi.Model(blob), n, nn_x=edge, nn_y=edge, precision=capi.PRECISION_FP16)
        out = h.forward(sp, gl)
        h.close()
        rows = [0, 1, n // 2, n - 2, n - 1]
        ref = oracle.OracleModel(blob, edge, edge).forward(sp[rows], gl[rows])
        for k in ref:
            got = out[k][rows]
            assert np.all(np.abs(got - ref[k]) <= 0.03 * np.maximum(np.maximum(np.abs(got), np.abs(ref[k])), 3.0)), (trunk, mid, k)


@pytest.mark.parametrize("d,heads,head_dim,ffn,rope", [(96, 3, 32, 160, "learnable"), (96, 2, 64, 96, "fixed"), (160, 5, 64, 416, "learnable"),
                                                        (224, 4, 64, 320, "none")])
@pytest.mark.parametrize("n", [3, 40])
def test_transformers_with_partial_chunks(d, heads, head_dim, ffn, rope, n, oracle):
    """Trunk and FFN widths that end inside a 64-channel chunk: the folded RMS norms, the rotary and the SwiGLU epilogues then run
    on the tensor-core path too.  Bounds as for the other transformers in reduced precision."""
    from tests.test_gpu_parity import _assert_reduced_close  # (not at the top: its tests would be collected here again)
    blob = mf.to_blob(mf.make_transformer(seed=470 + d, layers=2, d=d, heads=heads, head_dim=head_dim, ffn=ffn, rope=rope, rel_bias=rope == "none"))
    sp, gl = mf.random_positions(n, seed=15, board_sizes=([19, 13, 9] * n)[:n])
    h = capi.Handle(capi.Model(blob), n, precision=capi.PRECISION_FP16)
    out = h.forward(sp, gl)
    h.close()
    rows = list(range(3)) if n == 3 else [0, 1, 20, n - 2, n - 1]
    ref = oracle.OracleModel(blob).forward(sp[rows], gl[rows])
    _assert_reduced_close({k: v[rows] for k, v in out.items()}, ref, sp[rows][..., 0].reshape(len(rows), -1))


@pytest.mark.parametrize("trunk,mid", [(96, 528), (72, 640), (528, 96), (64, 576)])
def test_more_activated_channels_than_the_tensor_core_kernel_holds(trunk, mid, oracle):
    """The norm parameters of more than 512 channels do not fit that kernel: such a layer runs on the CUDA cores, at any input
    width.  Tolerance as above; once as a block and once in a net, whose first convolution and block ends are as wide."""
    g = mf._Gen(450 + trunk + mid)
    rng = np.random.default_rng(trunk + mid)
    mask = np.ones((2, 9, 9), np.float32)
    mask[1, 7:] = 0
    layer = mf._gen_ordinary(g, trunk, mid, mf.ACT_MISH)
    x = rng.standard_normal((2, 9, 9, trunk)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, trunk)
    out = capi.eval_layer(blob, x, mask, trunk, precision=capi.PRECISION_FP16)
    assert np.all(np.abs(out - ref) <= 0.03 * np.maximum(np.maximum(np.abs(out), np.abs(ref)), 3.0))
    blob = mf.to_blob(mf.make_convnet("wide", 451, 15, trunk, ["plain", "plain"], (32, 32, 32, 64), mf.ACT_MISH, mid_c=mid, regular_c=64, gpool_c=32))
    sp, gl = mf.random_positions(2, seed=9, nn_len=9)
    ref = oracle.OracleModel(blob, 9, 9).forward(sp, gl)
    h = capi.Handle(capi.Model(blob), 2, nn_x=9, nn_y=9, precision=capi.PRECISION_FP16)
    for _ in range(2):  # the eager run and the graph
        out = h.forward(sp, gl)
        for k in ref:
            assert np.all(np.abs(out[k] - ref[k]) <= 0.03 * np.maximum(np.maximum(np.abs(out[k]), np.abs(ref[k])), 3.0)), k
    h.close()


@pytest.mark.parametrize("factory,prec,full,edge", [
    (lambda: mf.make_b18c384nbt(num_blocks=3), capi.PRECISION_FP16, 128, 19),
    (lambda: mf.make_b18c384nbt(num_blocks=3), capi.PRECISION_BF16, 128, 9),
    (lambda: mf.make_b28c512nbt(num_blocks=3), capi.PRECISION_BF16, 128, 19),
    (lambda: mf.make_b28c512nbt(num_blocks=3), capi.PRECISION_FP16, 64, 13),
    (lambda: mf.make_b6c96(), capi.PRECISION_FP16, 256, 19),
    (lambda: mf.make_transformer(layers=2), capi.PRECISION_FP16, 64, 19),
    (lambda: mf.make_transformer_relbias(layers=2), capi.PRECISION_FP16, 64, 19),
    # widths that the small tiles do not divide, and a layer (96->288) that keeps to the wide ones among layers that do not
    (lambda: mf.make_convnet("tiles", 81, 15, 160, ["plain", "plain"], (32, 32, 32, 64), mf.ACT_MISH, mid_c=224, regular_c=64, gpool_c=32),
     capi.PRECISION_FP16, 128, 19),
    (lambda: mf.make_convnet("tiles", 82, 15, 320, ["plain", "gpool", "plain"], (32, 32, 32, 64), mf.ACT_MISH, mid_c=96, regular_c=64, gpool_c=32),
     capi.PRECISION_BF16, 128, 19),
    (lambda: mf.make_convnet("tiles", 83, 15, 288, ["plain", "plain"], (32, 32, 32, 64), mf.ACT_MISH, mid_c=96, regular_c=64, gpool_c=32),
     capi.PRECISION_FP16, 128, 19),
    # transformers of other widths: other wide tiles and warps behind the order of the row sums, and consumers of row sums without small
    # tiles (832 = 4 x 208 channels), whose producers then have none either
    (lambda: mf.make_transformer(layers=2, d=96, heads=3, head_dim=32, ffn=160), capi.PRECISION_FP16, 128, 19),
    (lambda: mf.make_transformer(layers=2, d=160, heads=5, head_dim=64, ffn=416), capi.PRECISION_FP16, 64, 19),
    (lambda: mf.make_transformer(layers=2, d=224, heads=4, head_dim=64, ffn=320, rope="none", rel_bias=True), capi.PRECISION_BF16, 64, 19),
    (lambda: mf.make_transformer(layers=2, d=512, heads=8, head_dim=64, ffn=1024, rope="fixed"), capi.PRECISION_FP16, 64, 13),
])
def test_small_batches_give_the_rows_of_a_full_batch(factory, prec, full, edge):
    """Small batches run in narrow tiles (kb_conv_small.cu), full ones in wide tiles and merged launches.  The order of an
    accumulator's additions depends on neither, so a position's outputs are the same bits whatever batch it is in."""
    model = capi.Model(mf.to_blob(factory()))
    h = capi.Handle(model, full, nn_x=edge, nn_y=edge, precision=prec)
    sizes = ([edge, 9, 7, edge] * full)[:full]
    sp, gl = mf.random_positions(full, seed=61, nn_len=edge, board_sizes=sizes)
    ref = h.forward(sp, gl)
    for n in (1, 2, 5, 11, 12, 13, 24, 25, 32, 48):
        for _ in range(2):  # the eager run and the graph
            part = h.forward(sp[:n], gl[:n])
            for k in ref:
                assert np.array_equal(part[k], ref[k][:n]), (n, k)
    h.close()


@pytest.mark.parametrize("make", [mf.make_transformer, mf.make_transformer_relbias])
@pytest.mark.parametrize("n", [1, 3])
def test_tile_dependencies_leave_row_sums_in_the_form_they_are_read(make, n, monkeypatch):
    """With KB_TILE_DEPS a convolution that reports its tiles runs in wide tiles in every batch: the row sums of its output then have to
    be read in the form of the wide tiles.  The same bits as without the switch."""
    model = capi.Model(mf.to_blob(make(layers=2)))
    sp, gl = mf.random_positions(n, seed=18, board_sizes=[19, 13, 9][:n])
    outs = {}
    for mode in ("0", "1", "2"):
        monkeypatch.setenv("KB_TILE_DEPS", mode)  # read when a handle is created
        h = capi.Handle(model, n, precision=capi.PRECISION_FP16)
        outs[mode] = [h.forward(sp, gl) for _ in range(3)]
        h.close()
    for mode in outs:
        for run in outs[mode]:
            for k in run:
                assert np.array_equal(run[k], outs["0"][0][k]), (mode, k)


@pytest.mark.parametrize("trunk,mid", [(512, 256), (256, 128), (128, 64), (320, 192), (384, 128), (192, 64)])
@pytest.mark.parametrize("prec", [capi.PRECISION_FP16, capi.PRECISION_BF16])
def test_fused_closing_and_opening_convolutions(trunk, mid, prec):
    """The fused 1x1 pair at every part width (64, 128, 192 channels), with one and two accumulators of its first GEMM and weights of
    the second in one or several pieces, at more tiles than SMs: the bits of separate launches."""
    blob = mf.to_blob(mf.make_nbt("pair", 3, 4, trunk, mid, 32, (32, 32, 64, 96)))
    n = 70
    sp, gl = mf.random_positions(n, seed=5, board_sizes=([19, 13, 9, 19] * n)[:n])
    outs = {}
    old = os.environ.get("KB_FUSE_1X1")
    try:
        for mode in ("0", "1"):
            os.environ["KB_FUSE_1X1"] = mode
            h = capi.Handle(capi.Model(blob), n, precision=prec)
            outs[mode] = [h.forward(sp, gl) for _ in range(3)]
            h.profile_enable(True)
            h.forward_resident(n)
            assert any("fused" in e["name"] and e["launches"] for e in h.profile_read()) == (mode == "1")
            h.close()
    finally:
        if old is None:
            os.environ.pop("KB_FUSE_1X1", None)
        else:
            os.environ["KB_FUSE_1X1"] = old
    for run in outs["0"] + outs["1"]:
        for k in run:
            assert np.array_equal(run[k], outs["0"][0][k]), k


def _locked(a, keep, shift=0):
    """A copy of `a` in page-locked memory, `shift` elements behind an aligned address."""
    flat = capi.PinnedArray((a.size + shift,), a.dtype)
    keep.append(flat)
    view = flat.array[shift:].reshape(a.shape)
    view[...] = a
    return view


@pytest.mark.parametrize("n", [1, 3, 60, 133])
def test_host_buffers_of_every_kind(n):
    """Page-locked buffers (moved by a kernel in small calls, with or without 16-byte alignment), pageable ones and a mixture of
    the two, and calls that leave outputs out: the same bits.  60 positions are past the limit of the kernel that reads, 133 past
    that of the one that writes too."""
    model = capi.Model(mf.to_blob(mf.make_b6c96()))
    h = capi.Handle(model, n, precision=capi.PRECISION_FP16)
    sp, gl = mf.random_positions(n, seed=17)
    sym = np.arange(n, dtype=np.int32) % 8
    ref = h.forward(sp, gl, sym)
    keep = []
    for shift in (0, 1):
        ins = [_locked(a, keep, shift) for a in (sp, gl, sym)]
        outs = {k: _locked(np.zeros_like(v), keep, shift) for k, v in ref.items()}
        for left_out in ((), ("policy", "value"), ("ownership",), tuple(ref)):
            for v in outs.values():
                v[...] = -1
            h.forward(*ins, out={k: None if k in left_out else v for k, v in outs.items()})
            assert all(np.all(outs[k] == -1) if k in left_out else np.array_equal(outs[k], ref[k]) for k in ref), left_out
    mixed = h.forward(sp, ins[1], ins[2], out={k: (outs[k] if k == "policy" else np.zeros_like(v)) for k, v in ref.items()})
    assert all(np.array_equal(mixed[k], ref[k]) for k in ref)
    h.close()


@pytest.mark.parametrize("n", [2, 60])
def test_page_locked_metadata_and_two_handles_at_once(n):
    """Metadata rows in page-locked memory, and two handles whose calls share the GPU from two threads: every call's own outputs."""
    model = capi.Model(mf.to_blob(mf.add_meta_encoder(mf.make_b6c96())))
    keep, states, errors = [], [], []
    for seed in (18, 19):
        h = capi.Handle(model, n, precision=capi.PRECISION_FP16)
        ins = mf.random_positions(n, seed=seed) + (np.arange(n, dtype=np.int32) % 8,)
        meta = mf.random_meta_rows(n, seed=seed, channels=model.meta_c)
        ref = h.forward(*ins, meta=meta)
        states.append((h, [_locked(a, keep) for a in ins], _locked(meta, keep), {k: _locked(np.zeros_like(v), keep) for k, v in ref.items()}, ref))

    def work(h, ins, meta, outs, ref):
        try:
            for _ in range(200):
                for v in outs.values():
                    v[...] = -1
                h.forward(*ins, out=outs, meta=meta)
                assert all(np.array_equal(outs[k], ref[k]) for k in ref)
        except Exception as e:  # handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=s) for s in states]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for s in states:
        s[0].close()


@pytest.mark.parametrize("prec,tol", [(capi.PRECISION_FP16, 0.03), (capi.PRECISION_BF16, 0.2)])
@pytest.mark.parametrize("trunk,mid", [(32, 32), (160, 224), (288, 96), (320, 96), (448, 160)])
@pytest.mark.parametrize("n", [1, 4, 7, 16, 31])
def test_tiles_that_end_inside_a_layer(prec, tol, trunk, mid, n, oracle):
    """Widths that the tiles of the small-batch kernel (32 to 192 channels, 64 or 128 rows) do not divide, at batches from its
    narrowest tiles to two CTAs per SM: the last tile of a row is short, the last row tile reaches into the padding.  (Of 288 and 96
    the layer to 288 keeps to the wide kernels, whose tile of 144 channels is no multiple of 32; its neighbour does not.)  Tolerance as
    in test_input_widths_between_chunks."""
    small = [capi.tile_plan(3, i, o)["bn"] % 32 == 0 for i, o in ((trunk, mid), (mid, trunk))]
    assert small == [True, trunk != 288]
    g = mf._Gen(700 + trunk + mid)
    rng = np.random.default_rng(trunk + mid + n)
    mask = np.ones((n, 19, 19), np.float32)
    mask[0, 13:] = 0
    layer = mf._gen_ordinary(g, trunk, mid, mf.ACT_MISH)
    x = rng.standard_normal((n, 19, 19, trunk)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, trunk)
    out = capi.eval_layer(blob, x, mask, trunk, precision=prec)
    assert np.all(np.abs(out - ref) <= tol * np.maximum(np.maximum(np.abs(out), np.abs(ref)), 3.0))


@pytest.mark.parametrize("trunk,mid", [(4, 8), (20, 36), (96, 96), (64, 100), (132, 48)])
@pytest.mark.parametrize("n,ylen,xlen", [(1, 19, 19), (5, 9, 13), (2, 5, 30)])
def test_fp32_block_widths(trunk, mid, n, ylen, xlen, oracle):
    """fp32 residual blocks at the edges of the staged kernel's tiles (16-channel slices, tiles of 32 channels and 32 to 80 rows, wide
    boards with their larger halo).  A sum of K products of order one in fp32 is off by at most about K * 2^-24 of their
    magnitude: 2 * 9 * 132 * 6e-8 = 1.4e-4 in the worst case and two orders less in practice; 1e-4 as for the other fp32 tests."""
    g = mf._Gen(500 + trunk + mid)
    rng = np.random.default_rng(trunk + 7 * mid)
    mask = np.ones((n, ylen, xlen), np.float32)
    mask[0, ylen // 2:] = 0
    layer = mf._gen_ordinary(g, trunk, mid, mf.ACT_MISH)
    x = rng.standard_normal((n, ylen, xlen, trunk)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, trunk)
    out = capi.eval_layer(blob, x, mask, trunk, precision=capi.PRECISION_FP32)
    assert np.abs(out - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("reg,gp", [(32, 8), (64, 16), (96, 64), (160, 32), (40, 128), (64, 24), (80, 48), (64, 192), (48, 320), (32, 1024)])
@pytest.mark.parametrize("n,edge", [(1, 19), (11, 9), (80, 13)])
def test_gpool_widths(reg, gp, n, edge, oracle):
    """Global-pooling blocks at the widths where the fused middle changes its split (channels per CTA, lanes per pooled
    channel) or adds up in another way (a number of 8-channel pieces that does not divide a warp), for few and for many boards; the tolerance is the
    reference's reduced-precision layer tolerance (cpp/tests/testnn.cpp:8-15)."""
    C = 64
    g = mf._Gen(600 + reg + gp)
    rng = np.random.default_rng(reg * gp + n)
    mask = np.ones((n, edge, edge), np.float32)
    mask[0, :, edge // 2:] = 0
    layer = mf._gen_gpool(g, C, reg, gp, mf.ACT_MISH)
    x = rng.standard_normal((n, edge, edge, C)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, C)
    out = capi.eval_layer(blob, x, mask, C, precision=capi.PRECISION_FP16)
    assert np.all(np.abs(out - ref) <= 0.03 * np.maximum(np.maximum(np.abs(out), np.abs(ref)), 3.0))


@pytest.mark.parametrize("gp", [24, 40, 48, 96, 192, 512])
def test_gpool_middle_is_one_launch(gp):
    """Every pooled width that is a multiple of 8 takes the fused middle."""
    def launches(gp):
        tree = mf.make_convnet("gp", 610, 15, 64, ["gpool"], (32, 32, 32, 64), mf.ACT_RELU, regular_c=64, gpool_c=gp)
        h = capi.Handle(capi.Model(mf.to_blob(tree)), 4, nn_x=9, nn_y=9, precision=capi.PRECISION_FP16)
        n = h.launches_per_forward(4)
        h.close()
        return n
    assert launches(gp) == launches(32)


@pytest.mark.parametrize("n", [3, 44])
def test_gpool_middle_with_more_than_48_kb(n, oracle):
    """How many channels a CTA of the fused middle takes, and with them its shared memory, grows with the number of boards: past
    42 boards these widths need 49 KB.  Tolerance as above."""
    C, reg, gp = 16, 3584, 256
    g = mf._Gen(620)
    rng = np.random.default_rng(n)
    mask = np.ones((n, 5, 5), np.float32)
    mask[0, 3:] = 0
    layer = mf._gen_gpool(g, C, reg, gp, mf.ACT_MISH)
    x = rng.standard_normal((n, 5, 5, C)).astype(np.float32) * mask[..., None]
    blob = mf.layer_blob(layer)
    ref = oracle.eval_layer(blob, x, mask, C)
    out = capi.eval_layer(blob, x, mask, C, precision=capi.PRECISION_FP16)
    assert np.all(np.abs(out - ref) <= 0.03 * np.maximum(np.maximum(np.abs(out), np.abs(ref)), 3.0))


def test_head_kernels_of_different_sizes_from_two_threads(monkeypatch):
    """The fused heads need more shared memory than a kernel has by default for wide heads, and how much depends on the net: two
    nets that are run from two threads must not take the larger limit away from each other."""
    monkeypatch.setenv("KB_NO_GRAPH", "1")  # read when a handle is created: every pass launches its kernels anew
    sp, gl = mf.random_positions(1, seed=12, nn_len=5)
    handles, refs, errors = [], [], []
    for seed, g1 in ((900, 408), (901, 448)):
        tree = mf.make_convnet("heads", seed, 15, 64, ["plain"], (512, g1, 64, 64), mf.ACT_RELU, regular_c=32, gpool_c=32)
        handles.append(capi.Handle(capi.Model(mf.to_blob(tree)), 1, nn_x=5, nn_y=5, precision=capi.PRECISION_FP16))
        refs.append(handles[-1].forward(sp, gl))

    def work(h, ref):
        try:
            for _ in range(3000):
                out = h.forward(sp, gl)
                assert all(np.array_equal(out[k], ref[k]) for k in ref)
        except Exception as e:  # handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(handles, refs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for h in handles:
        h.close()


def test_profile_counts_what_a_small_batch_launches():
    """A small batch runs the members of merged launches one by one: the profile has them under their own names, with their own
    bytes, and as many as the launch count says; a full batch has the merged launches."""
    h = capi.Handle(capi.Model(mf.to_blob(mf.make_b18c384nbt(num_blocks=3))), 128, precision=capi.PRECISION_FP16)
    sp, gl = mf.random_positions(128, seed=13)
    h.upload(sp, gl)
    h.profile_enable(True)
    totals = {}
    for n in (2, 128):
        h.profile_reset()
        h.forward_resident(n)
        ran = [e for e in h.profile_read() if e["launches"]]
        assert sum(e["launches"] for e in ran) == h.launches_per_forward(n)
        assert any("chain" in e["name"] or "fused" in e["name"] for e in ran) == (n == 128)
        totals[n] = (sum(e["flops"] for e in ran) / n, sum(e["bytes"] for e in ran) / n)
    h.close()
    assert totals[2][0] == pytest.approx(totals[128][0])
    assert totals[2][1] > totals[128][1]  # the activated trunk tensor, which the fused 1x1 launches do not write


def test_both_forms_of_the_bounded_wait_give_up():
    """Those of feeding and issuing warps, and the plain one.  199 is the time-out itself; 198 would be a wait that reported success or
    recorded nothing, or a slot armed again behind a failed one."""
    h = capi.Handle(capi.Model(mf.to_blob(mf.make_b18c384nbt(num_blocks=1))), 1, precision=capi.PRECISION_FP16)
    with pytest.raises(capi.KBError, match="status 199:"):
        h.selftest_wait_timeout(1_000_000)
    h.close()


def test_noalloc_convolution_after_another_geometry(oracle):
    """kb_conv_noalloc keeps one buffer for all geometries: a call's padding rows may hold an earlier call's board points, in
    widths that the engine's staged fp32 kernel would take."""
    pytest.importorskip("torch")
    from tests.test_zz_no_alloc import _run_pair
    import torch
    g = mf._Gen(77)
    rng = np.random.default_rng(3)
    for n, ylen, xlen in [(3, 19, 19), (2, 7, 30), (4, 9, 9), (1, 19, 19)]:
        _run_pair(torch, g.conv(3, 64, 32), rng.standard_normal((n, ylen, xlen, 64)).astype(np.float32), oracle)
