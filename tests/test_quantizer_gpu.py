"""GPU parity of the load-time MXFP4 quantiser (byte work: bit-exact) and of loading a layer from fp32."""
import os

import numpy as np
import pytest

from conftest import GOLDEN_DIR

pytestmark = pytest.mark.gpu


def gpu_quantize(pkg, vals):
    import torch
    n = vals.size
    nblk = (n + 31) // 32
    d_v = torch.from_numpy(np.ascontiguousarray(vals, dtype=np.float32)).cuda()
    d_c = torch.full((nblk * 16,), 0xAB, dtype=torch.uint8, device="cuda")
    d_s = torch.full((nblk,), 0xCD, dtype=torch.uint8, device="cuda")
    pkg.quantize_mxfp4(d_v.data_ptr(), n, d_c.data_ptr(), d_s.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return d_c.cpu().numpy(), d_s.cpu().numpy()


def test_quantizer_golden_edge_cases(pkg, synth):
    z = np.load(os.path.join(GOLDEN_DIR, "quant_edge_cases.npz"))
    codes, scales = gpu_quantize(pkg, z["values"])
    assert np.array_equal(scales, z["scales"])
    assert np.array_equal(codes, z["codes"])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4096, 32 * 5000 + 17])
def test_quantizer_matches_oracle(n, pkg, port):
    rng = np.random.default_rng(n)
    v = (rng.standard_normal(n) * np.exp(rng.uniform(-25, 25, n))).astype(np.float32)
    if n >= 4096:
        v[64:96] = 0.0
        v[200] = np.nan                      # a NaN never becomes the block maximum and encodes as code 0
    pc, ps = port.quantize(v)
    gc, gs = gpu_quantize(pkg, v)
    assert np.array_equal(gs, ps) and np.array_equal(gc, pc)


@pytest.mark.parametrize("src_offset", [0, 1])
def test_quantizer_midpoints_and_neighbours(src_offset, pkg, port):
    """Every magnitude and midpoint of the table, one and two last places to either side, both signs, under block
    maxima of several exponents (the smallest ones on the library-call path), zeros and NaN between them."""
    grid = np.array([0.0, 0.125, 0.25, 0.5, 0.75, 1.0, 1.25, 1.5, 1.75, 2.0, 2.5, 3.0, 3.5, 4.0, 5.0, 6.0, 7.0],
                    dtype=np.float32)
    near = np.concatenate([grid, np.nextafter(grid, np.float32(9)), np.nextafter(grid, np.float32(-9)),
                           np.nextafter(np.nextafter(grid, np.float32(9)), np.float32(9))])
    near = np.concatenate([near, -near])
    blocks = []
    for e in (-126, -125, -122, -60, -7, 0, 30, 120):
        for i in range(0, len(near), 30):
            b = np.zeros(32, np.float32)
            part = near[i:i + 30]
            b[1:1 + len(part)] = part
            b[0] = 4.0 if i % 60 else -7.9375      # sets the block's exponent
            b[31] = np.nan if i == 30 else 0.0
            blocks.append(b * np.float32(2.0) ** np.float32(e))
    v = np.concatenate([np.zeros(src_offset, np.float32)] + blocks)[src_offset:]
    pc, ps = port.quantize(v)
    import torch
    d_v = torch.zeros(v.size + src_offset, dtype=torch.float32, device="cuda")
    d_v[src_offset:] = torch.from_numpy(v).cuda()   # offset 1: the scalar-load path
    d_c = torch.empty(v.size // 2, dtype=torch.uint8, device="cuda")
    d_s = torch.empty(v.size // 32, dtype=torch.uint8, device="cuda")
    pkg.quantize_mxfp4(d_v[src_offset:].data_ptr(), v.size, d_c.data_ptr(), d_s.data_ptr(),
                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(d_s.cpu().numpy(), ps) and np.array_equal(d_c.cpu().numpy(), pc)


def test_quantizer_full_size_properties(pkg, synth, port):
    """One expert's MLP1 matrix at full size (5760 x 2880 fp32, 66 MB): quantising the exact decode of
    MXFP4 weights gives back values that decode to the same floats (a block whose largest code is 3 or
    less moves to the next lower scale; its values stay representable), and the scales never exceed the
    original ones."""
    layer = synth.make_layer(1, 2880, 2880, seed=5)
    w = synth.dequant_mxfp4(layer["w1_codes"][0], layer["w1_scales"][0]).astype(np.float32)
    gc, gs = gpu_quantize(pkg, w.reshape(-1))
    back = port.dequant(gc.reshape(-1, 16), gs.reshape(-1, 1)).reshape(w.shape)
    assert np.array_equal(back, w)
    assert (gs.reshape(layer["w1_scales"][0].shape) <= layer["w1_scales"][0]).all()


def test_load_layer_f32_equals_load_layer(pkg, synth):
    """A layer loaded from the fp32 decode of its MXFP4 tensors gives the same output bits."""
    E, H, D, T = 8, 128, 160, 50
    layer = synth.make_layer(E, H, D, seed=33)
    tokens = synth.make_tokens(T, H, seed=34)
    a = pkg.MoeBlock(H, D, E, max_rows=T)
    b = pkg.MoeBlock(H, D, E, max_rows=T)
    try:
        a.load_layer(0, layer)
        w1 = synth.dequant_mxfp4(layer["w1_codes"], layer["w1_scales"])
        w2 = synth.dequant_mxfp4(layer["w2_codes"], layer["w2_scales"])
        b.load_layer_f32(0, w1, synth.bf16_bits_to_f32(layer["b1"]), w2, synth.bf16_bits_to_f32(layer["b2"]),
                         layer["router_w"], layer["router_b"])
        assert np.array_equal(a.forward_host(0, tokens), b.forward_host(0, tokens))
    finally:
        a.close()
        b.close()
