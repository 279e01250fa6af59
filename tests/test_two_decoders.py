"""Two decoders that step side by side on one GPU: what one computes does not depend on what else the GPU is doing. The
other decoder's kernels slow down parts of a kernel against one another by microseconds, which its hand-overs between
warps, copies and tensor cores have to allow for."""

import functools
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
STEPS = 100


@functools.lru_cache(maxsize=1)
def _model():
    from cohere_inference_b200.synth import synthetic_model
    return synthetic_model(3, layers=2, bias_std=0.05).cuda()


def _decoder(rows, kw):
    from cohere_inference_b200 import StreamDecoder
    return StreamDecoder(_model(), slots=rows, buckets=(rows,), max_new_tokens=8, max_prompt=STEPS, max_audio_s=30.0,
                         eos=-1, record=True, **kw)


def _admit(dec, rows, seed):
    """`rows` seeded requests whose prompts are fed for all the steps; returns the bucket."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(1, 376, rows).tolist()
    memory = torch.from_numpy(rng.standard_normal((sum(lens), 1024)).astype(np.float32)).cuda()
    dec.reset()
    with torch.cuda.stream(dec.stream):
        dec.fill_cross(memory, lens, list(range(rows)))
    dec.admit(list(range(rows)), [torch.from_numpy(rng.integers(0, 16384, STEPS)) for _ in lens], lens)
    bucket = dec.set_active(list(range(rows)))
    torch.cuda.synchronize()
    return bucket


def _steps(dec, rows, bucket):
    """Per step, row and vocabulary tile: the sum of the logits (the same bits for the same logits)."""
    out = torch.zeros(STEPS, rows, 128, device="cuda")
    with torch.cuda.stream(dec.stream):
        dec.stream.wait_stream(torch.cuda.default_stream())
        for t in range(STEPS):
            dec.step(bucket)
            out[t].copy_(dec.logits[:rows].view(rows, 128, 128).double().sum(-1).float())
    dec.check_status()
    return out.cpu().numpy()


@pytest.mark.parametrize("first,second", [
    ((24, dict(int8=True)), (24, dict(int8=True))),
    ((64, dict(int8=True)), (64, dict(int8=True))),
    ((128, dict(int8=True)), (48, dict(int8=True))),
    ((64, dict(int8=True, ffn_sparse=True)), (32, dict(fp16_weights=True))),
    ((32, dict(int8=True, attn_ring=True)), (32, dict(int8=True, attn_ring=True))),
    ((12, dict(int8=True, kv_int8=True)), (24, dict())),
])
def test_a_decoder_beside_another_gives_the_bits_it_gives_alone(first, second):
    sides = [(_decoder(*s), s[0]) for s in (first, second)]
    alone = [_steps(d, rows, _admit(d, rows, i)) for i, (d, rows) in enumerate(sides)]
    for _ in range(2):
        buckets = [_admit(d, rows, i) for i, (d, rows) in enumerate(sides)]
        got = [None, None]

        def serve(i):
            got[i] = _steps(*sides[i], buckets[i])
        threads = [threading.Thread(target=serve, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i in range(2):
            assert np.array_equal(got[i], alone[i]), (i, np.argwhere(got[i] != alone[i])[:8])


@pytest.mark.parametrize("rows,kw", [(8, dict(int8=True)), (24, dict(int8=True)), (64, dict(int8=True, kv_int8=True)),
                                     (24, dict(fp16_weights=True)), (8, dict())])
def test_steps_and_prefills_side_by_side_give_their_bits(rows, kw):
    """Clips that are admitted while others decode: their prefill runs on a stream of its own beside the steps in flight,
    as DecodeScheduler has it."""
    from cohere_inference_b200 import StreamDecoder
    dec = StreamDecoder(_model(), slots=rows + 8, buckets=(rows,), max_new_tokens=8, max_prompt=STEPS, max_audio_s=30.0,
                        eos=-1, record=True, **kw)
    names = ["cross_k", "cross_v"] + (["cross_ks", "cross_vs"] if kw.get("kv_int8") else [])
    lens, slots = [375, 300, 77, 1, 129, 250, 375, 33], list(range(rows, rows + 8))
    g = torch.Generator(device="cuda").manual_seed(1)
    clips = [torch.randn(sum(lens), 1024, device="cuda", generator=g).to(t) for t in (torch.float32, torch.bfloat16)]

    def caches():
        return [torch.cat([getattr(dec, n)[:, s, :, :f].flatten() for s, f in zip(slots, lens)]) for n in names]
    want = []
    for x in clips:
        with torch.cuda.stream(dec.stream):
            dec.stream.wait_stream(torch.cuda.default_stream())
            dec.fill_cross(x, lens, slots)
        dec.check_status()
        want.append(caches())
    alone = _steps(dec, rows, _admit(dec, rows, 0))
    bucket, got, stop, fills = _admit(dec, rows, 0), [], threading.Event(), [0]

    def serve():
        got.append(_steps(dec, rows, bucket))
        stop.set()
    t = threading.Thread(target=serve)
    side = torch.cuda.Stream()
    t.start()
    while not stop.is_set() or fills[0] < 2:
        i = fills[0] % 2
        with torch.cuda.stream(side):
            dec.fill_cross(clips[i], lens, slots)
            now = caches()
        side.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(now, want[i]))
        fills[0] += 1
    t.join()
    assert np.array_equal(got[0], alone)
