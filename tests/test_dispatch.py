"""Which kernel a size goes to: the rules of kernels/ops.py, checked without a GPU."""
import torch

from photon_infer_b200.kernels import ops


def test_tcgen05_product_wants_enough_tiles_and_rows():
    assert ops.gemm_tc_tiles(64, 3072) == 0                       # a tile of 128 rows would be mostly padding
    assert ops.gemm_tc_tiles(128, 3072) == 12
    assert ops.gemm_tc_tiles(2048, 3072) == 16 * 12
    assert ops.gemm_tc_tiles(2048, 16384, swiglu=True) == 16 * 64  # a SwiGLU tile covers 128 output columns
    assert ops.gemm_tc_tiles(512, 3072) < ops.TC_MIN_TILES <= ops.gemm_tc_tiles(2048, 2048)
    assert ops.TC_PAIR_MIN_ROWS == 256 and ops.SKINNY_MAX_ROWS == 8


def test_tcgen05_product_refuses_what_tma_cannot_load():
    x = torch.zeros(256, 64, dtype=torch.bfloat16)
    w = torch.zeros(512, 64, dtype=torch.bfloat16)
    assert ops.gemm_tc_supported(x, w)
    assert not ops.gemm_tc_supported(x.float(), w.float())        # bfloat16 only
    assert not ops.gemm_tc_supported(x[:, :60], w[:, :60])        # K not a multiple of 8, rows not contiguous
    assert not ops.gemm_tc_supported(x, w[::2])                   # weight not contiguous
    xs = torch.zeros(256, 72, dtype=torch.bfloat16)[:, :64]       # row stride 72: a multiple of 8, allowed
    assert ops.gemm_tc_supported(xs, w)
    xo = torch.zeros(256 * 64 + 4, dtype=torch.bfloat16)[4:].view(256, 64)   # base 8 bytes off a 16-byte boundary
    assert not ops.gemm_tc_supported(xo, w)


def test_qkv_epilogue_wants_long_portions_and_heads_in_steps_of_32():
    w = torch.zeros(3072, 2048, dtype=torch.bfloat16)
    assert ops.gemm_tc_qkv_supported(torch.zeros(2048, 2048, dtype=torch.bfloat16), w, 64)
    assert ops.gemm_tc_qkv_supported(torch.zeros(2048, 2048, dtype=torch.bfloat16), w, 128)
    assert not ops.gemm_tc_qkv_supported(torch.zeros(2048, 2048, dtype=torch.bfloat16), w, 48)
    assert not ops.gemm_tc_qkv_supported(torch.zeros(128, 2048, dtype=torch.bfloat16), w, 64)    # fewer than 256 rows
    assert not ops.gemm_tc_qkv_supported(torch.zeros(512, 2048, dtype=torch.bfloat16), w, 64)    # too few tiles


def test_tcgen05_attention_sizes():
    bf = torch.bfloat16
    for group in (1, 3, 4, 5, 128):
        assert ops.attention_tc_supported(bf, 64, group, 16)
    for page in (8, 16, 32, 64, 128, 256):
        assert ops.attention_tc_supported(bf, 128, 4, page)
    assert not ops.attention_tc_supported(bf, 64, 129, 16)        # more rows per token than a tile holds
    assert ops.attention_tc_supported(bf, 96, 4, 16) and ops.attention_tc_supported(bf, 40, 4, 16, 88)     # zeros behind the head
    assert not ops.attention_tc_supported(bf, 92, 4, 16)          # heads and values are multiples of 8 ..
    assert not ops.attention_tc_supported(bf, 64, 4, 16, 136)     # .. of at most 128
    assert not ops.attention_tc_supported(bf, 64, 4, 4)           # a TMA box needs pages of 8 tokens or more
    assert not ops.attention_tc_supported(bf, 64, 4, 24)          # pages must divide 64 or be a multiple of it
    assert not ops.attention_tc_supported(bf, 64, 4, 96)
    assert not ops.attention_tc_supported(torch.float32, 64, 4, 16)
    assert ops.flash_attention_supported(bf, 48) and not ops.flash_attention_supported(bf, 136)
    assert not ops.flash_attention_supported(torch.float32, 64)   # float32 takes the general kernel


def test_weight_streaming_product_sizes():
    x = torch.zeros(8, 2048, dtype=torch.bfloat16)
    w = torch.zeros(3072, 2048, dtype=torch.bfloat16)
    assert ops.skinny_gemm_supported(x, w)
    assert ops.skinny_gemm_supported(torch.zeros(64, 2048, dtype=torch.bfloat16), w)
    assert not ops.skinny_gemm_supported(torch.zeros(65, 2048, dtype=torch.bfloat16), w)
    assert not ops.skinny_gemm_supported(torch.zeros(33, 2048, dtype=torch.bfloat16), w, swiglu=True)
    assert not ops.skinny_gemm_supported(torch.zeros(8, 2044, dtype=torch.bfloat16), torch.zeros(16, 2044, dtype=torch.bfloat16))


def test_the_delta_rule_chooses_per_request():
    """What a request is run by depends on its own tokens; the long requests of a step together say whether there is enough work."""
    assert ops.delta_chunked_from(128, 128, [256] + [1] * 31, 32) == ops.DELTA_CHUNKED_MIN_TOKENS
    assert ops.delta_chunked_from(128, 128, [64] + [1] * 200, 32) == 0           # the decoded tokens are no work for the chunks
    assert ops.delta_chunked_from(128, 128, [63] * 100, 32) == 0
    assert ops.delta_chunked_from(129, 128, [4096], 32) == 0 and ops.delta_chunked_from(128, 257, [4096], 32) == 0


def test_segments_are_the_shortest_whose_long_requests_fit_at_once():
    """.. whatever stands beside the long requests, as long as that does not fill the GPU for their time."""
    import random
    rng = random.Random(1)
    for _ in range(2000):
        longs = [rng.randint(128, 4096) for _ in range(rng.choice((1, 1, 2, 3, 5, 9)))]
        heads, blocks = rng.choice((1, 2, 4, 8, 16, 32)), rng.choice((1, 2, 4))
        places, seg = max(1, 296 // (heads * blocks)), ops.linrec_segment_tokens(longs, heads, blocks, 148)
        cut = lambda n: sum(-(-x // n) for x in longs)
        assert seg % 16 == 0 and seg >= 64
        if places <= len(longs):
            assert cut(seg) == len(longs)                # as many segments as requests: nothing is cut
        else:
            assert cut(seg) <= places and (seg == 64 or cut(seg - 16) > places)
        others = [rng.randint(0, 127) for _ in range(rng.randint(0, 70))]
        mixed = longs + others
        rng.shuffle(mixed)
        rounds = len(others) * heads * blocks / 296
        want = -(-max(longs) // 16) * 16 if max(longs) <= ops.LINREC_SEGMENTS_BESIDE * rounds else seg
        assert ops.linrec_segment_tokens(mixed, heads, blocks, 148) == want
    assert ops.linrec_segment_tokens([2048] + [1] * 63, 16, 2, 148) == 240
    assert ops.linrec_segment_tokens([512] + [1] * 63, 32, 2, 148) == 512 and ops.linrec_segment_tokens([768] + [1] * 63, 32, 2, 148) == 192
    assert ops.linrec_segment_tokens([5, 90], 16, 2, 148) == 64


def test_the_switch_of_dependent_launches_takes_every_word_for_off(tmp_path):
    """``PHOTON_PDL``: unset, empty and 1 leave the launches on, everything else turns them off."""
    import os
    import subprocess

    from photon_infer_b200.csrc.build import CSRC_DIR, INCLUDE_DIR, find_nvcc
    src, exe = tmp_path / "pdl.cu", tmp_path / "pdl"
    src.write_text('#include "common.cuh"\n#include <cstdio>\nint main() { printf("%d", (int)photon_pdl_enabled()); return 0; }\n')
    subprocess.run([find_nvcc(), "-std=c++17", "-I", CSRC_DIR, "-I", INCLUDE_DIR, "-o", str(exe), str(src)], check=True, capture_output=True)
    env = {k: v for k, v in os.environ.items() if k != "PHOTON_PDL"}
    said = lambda value: subprocess.run([str(exe)], env=dict(env, PHOTON_PDL=value), capture_output=True, text=True).stdout
    assert subprocess.run([str(exe)], env=env, capture_output=True, text=True).stdout == "1"
    assert [said(v) for v in ("", "1", "0", "off", "no", "false")] == ["1", "1", "0", "0", "0", "0"]


def test_what_a_step_can_launch_is_built_at_load(monkeypatch):
    """The kernels that attention's 32-bit portions go to are among the modules that a model compiles before its first step, and are
    not where no step can go to them."""
    from photon_infer_b200.parts.attention import PagedAttention
    from photon_infer_b200.parts.normed_attention import NormedAttention

    class Taken(Exception):
        pass

    def taken(*args, **kwargs):
        raise Taken

    monkeypatch.setattr(ops, "attention_rows", taken)
    monkeypatch.setattr(ops, "paged_attention", lambda *args, **kwargs: None)
    part = lambda cls, *heads, **k: cls(256, *heads, **(dict(k, eps=1e-5) if cls is NormedAttention else k))
    for cls, extras in ((PagedAttention, ({}, {"window": 16})),
                        (NormedAttention, ({}, {"window": 16}, {"window": 16, "keep_first": 2}, {"sink": True}, {"softcap": 30.0}, {"output_gate": True},
                                           {"value_dim": 32}))):
        for heads in ((4, 2, 64), (32, 1, 128), (33, 1, 64), (4, 2, 96)):
            for extra in extras:
                mixer = part(cls, *heads, **extra)
                n_q, n_kv, d = heads
                v = getattr(mixer, "value_dim", d)
                q, out = torch.zeros(256, n_q * d), torch.zeros(256, n_q * v)
                if getattr(mixer, "sink", False):
                    mixer.sinks = torch.zeros(n_q)
                gate = torch.zeros(256, n_q * v) if extra.get("output_gate") else None
                ctx = type("Ctx", (), dict(max_query_len=256, num_seqs=1, num_tokens=256, cu_tokens=None, positions=None, token_seq=None,
                                           error_flag=None, max_context_len=256, groups=[type("G", (), dict(block_table=None))]))
                cache = type("C", (), dict(group=0, k=torch.zeros(4, n_kv, 16, d), v=torch.zeros(4, n_kv, 16, v)))
                try:
                    mixer.attend(q, out, ctx, cache, *([gate] if gate is not None else []))
                    goes = False
                except Taken:
                    goes = True
                assert goes == ("attention_rows" in mixer.required_kernels(torch.float32)), (cls, heads, extra)
                assert "attention_rows" not in mixer.required_kernels(torch.bfloat16)
