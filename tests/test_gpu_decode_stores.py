"""The segment decoder's staged words and 16-byte stores: segments starting at
every 4-byte offset, lengths around its 128-value blocks, and one longer than
its shared buffer, for every codec, against the encoded values."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("codec", range(1, 14))
def test_offsets_and_lengths(genie, codec):
    import torch
    lib = genie.lib()
    rng = np.random.default_rng(codec)
    lens = [1, 3, 127, 128, 129, 130, 255, 256, 257, 384, 511, 640, 1021, 1024, 5000]
    segs, vals, at, out_off = [], [], 0, []
    for shift in range(4):
        for n in lens:
            gap = rng.integers(0, 1 << int(rng.integers(1, 14)), n)
            v = np.cumsum(gap).astype(np.uint32)
            if codec == 3 and n % 2:
                v = rng.integers(0, 1 << 32, n, dtype=np.uint32)      # 32-bit widths
            buf = np.zeros(int(lib.genie_codec_encode_bound(n)) + 8, np.uint32)
            w = lib.genie_codec_encode(codec, v.ctypes.data, n, buf.ctypes.data, len(buf))
            assert w > 0
            segs.append(buf[:w].copy())
            vals.append(v)
            at += (shift - at) % 4
            out_off.append(at)
            at += n
    woff = np.concatenate([[0], np.cumsum([len(s) for s in segs])]).astype(np.int64)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    words, d_woff, d_off = dev(np.concatenate(segs).view(np.int32)), dev(woff), dev(np.array(out_off, np.int64))
    out = torch.full((at + 8,), -1, dtype=torch.int32, device="cuda")
    got_len = torch.zeros(len(segs), dtype=torch.int32, device="cuda")
    genie._check(lib.genie_codec_decode_device(codec, words.data_ptr(), d_woff.data_ptr(), len(segs), d_off.data_ptr(),
                                               out.data_ptr(), got_len.data_ptr(), ctypes.c_void_p(None)))
    torch.cuda.synchronize()
    expect = np.full(at + 8, 0xFFFFFFFF, np.uint32)
    for o, v in zip(out_off, vals):
        expect[o:o + len(v)] = v
    assert np.array_equal(got_len.cpu().numpy(), [len(v) for v in vals])
    assert np.array_equal(out.cpu().numpy().view(np.uint32), expect)
