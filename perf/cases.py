"""The work a program has this decoder do, as measurable cases.

Every case is one call (or one short sequence of calls) of the package's public
entry points on inputs made from a seed:

  tensor    cuopus_native.decode_ogg_to_cuda_tensor, one mono file -> float32 16 kHz
  multi     cuopus_native.decode_ogg_multi, several mono files in one launch
  channels  cuopus_native.decode_ogg_to_f16k_channels, mono or stereo files
  int16     cuopus_native.decode_ogg_to_int16, mono and stereo files -> int16 48 kHz
  batch     cuopus_native.decode_batch, the device-resident engine on whole streams
            (one chain per stream, work queue, longest first), optionally with lost
            packets and in-band FEC
  serve     serving.Server: requests submitted together, outputs read back to host
  resample  cuopus_resample48to16 on device-resident int16 PCM
  order     the learned scheduler's per-batch call: chain features + predictions

Opus packets come from the encoded streams under tests/golden/streams (made by the
libopus 1.5.2 encoder: SILK, hybrid and CELT, 2.5 to 120 ms packets, mono and
stereo).  A file is a splice of runs of 0.5-3 s taken from them at seeded places,
so modes switch every 0.5-3 s as in the mixed benchmark corpus, and is wrapped in
Ogg pages with valid checksums.  File lengths are the case's own (log-uniform
quantiles between min_s and max_s), so a case's work does not depend on the seed;
the seed picks the packets.
"""
import math
import os
import struct
import zlib

import numpy as np
import torch

from cuopus_b200 import cuopus_native as cn
from cuopus_b200 import costmodel, serving

GOLD = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "streams")
# content -> (source streams, channels of the file, about how many packet bytes a second)
CONTENT = {
    "voice": (("plain_a", "plain_b"), 1, 2500),                          # SILK wideband, 20 ms
    "speech": (("long_hybrid", "plain_b"), 1, 3200),                     # hybrid / SILK, 20 ms
    "mixed": (("mixed_mono_a", "mixed_mono_b", "long_hybrid", "code3_120ms"), 1, 3300),
    "stereo": (("mixed_stereo_a", "mixed_stereo_b"), 2, 6000),           # CELT / hybrid / SILK, stereo
}
F32_CALLS = ("tensor", "multi", "channels")


def listed():
    return [
        # a voice prompt or notification: one short file, pure latency
        {"name": "clip_0.4s", "call": "tensor", "content": "voice", "files": 1, "min_s": 0.4, "max_s": 0.4},
        # the plain benchmark shape: 64 one-second voice clips in one launch
        {"name": "voice_64x1s", "call": "multi", "content": "voice", "files": 64, "min_s": 1.0, "max_s": 1.0},
        # a voice memo or call recording, odd length
        {"name": "file_93.7s", "call": "tensor", "content": "mixed", "files": 1, "min_s": 93.7, "max_s": 93.7},
        # the long-file benchmark shape: 2 h of hybrid / SILK speech
        {"name": "long_7200s", "call": "tensor", "content": "speech", "files": 1, "min_s": 7200.0, "max_s": 7200.0},
        # a folder of stereo music and speech files to float32 at 16 kHz
        {"name": "stereo_f16k_12", "call": "channels", "content": "stereo", "files": 12, "min_s": 5.0, "max_s": 60.0},
        # a data loader's batch of files, mono and stereo, to int16
        {"name": "int16_30_files", "call": "int16", "content": "both", "files": 30, "min_s": 5.0, "max_s": 120.0},
        # the mixed-mode uneven batch, whole streams, device-resident
        {"name": "batch_512", "call": "batch", "content": "both", "files": 512, "min_s": 1.0, "max_s": 8.0,
         "loss": 0.0, "fec": 0},
        # the same engine on call audio with 5 % of the packets lost and in-band FEC
        {"name": "batch_loss_96", "call": "batch", "content": "mixed", "files": 96, "min_s": 0.5, "max_s": 3.0,
         "loss": 0.05, "fec": 1},
        # requests arriving together at the continuous-batching server
        {"name": "serve_24", "call": "serve", "content": "both", "files": 24, "min_s": 5.0, "max_s": 60.0},
        # the resampler alone, on an hour of device-resident PCM (odd length)
        {"name": "resample_1h", "call": "resample", "samples": 172800001},
        # visiting order of 4096 chains by the learned cost model
        {"name": "order_4096", "call": "order", "content": "both", "files": 4096, "min_s": 0.5, "max_s": 2.0},
    ]


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    """One more case of the ranges above; none costs more than the largest listed one."""
    call = rng.choice(["tensor", "tensor", "multi", "channels", "int16", "batch", "batch", "serve", "resample", "order"])
    if call == "resample":
        return {"call": call, "samples": int(_log_uniform(rng, 1000, 172800000)) | 1}
    if call == "tensor":
        s = round(_log_uniform(rng, 0.1, 3600.0), 2)
        return {"call": call, "content": rng.choice(["voice", "speech", "mixed"]), "files": 1, "min_s": s, "max_s": s}
    if call == "order":
        return {"call": call, "content": rng.choice(["mixed", "stereo", "both"]),
                "files": int(_log_uniform(rng, 16, 4096)), "min_s": 0.5, "max_s": 2.0}
    lo = round(_log_uniform(rng, 0.2, 5.0), 2)
    if call == "multi":
        return {"call": call, "content": rng.choice(["voice", "speech", "mixed"]), "files": rng.randint(2, 64),
                "min_s": lo, "max_s": round(lo * rng.uniform(1.0, 12.0), 2)}
    if call == "batch":
        lo = min(lo, 1.0)
        loss = rng.choice([0.0, 0.0, 0.02, 0.1])
        # every lost packet is 120 ms of concealment: fewer, shorter streams of 20 ms packets and longer
        content, most, longest = (["voice", "mixed"], 128, 3.0) if loss else (["voice", "mixed", "stereo", "both"], 512, 8.0)
        return {"call": call, "content": rng.choice(content), "files": int(_log_uniform(rng, 8, most)), "min_s": lo,
                "max_s": round(lo + (longest - lo) * rng.random(), 2), "loss": loss,
                "fec": int(loss > 0 and rng.random() < 0.7)}
    return {"call": call, "content": rng.choice(["mixed", "stereo", "both"]) if call != "channels" else
            rng.choice(["stereo", "stereo", "both"]), "files": rng.randint(1, 24), "min_s": lo,
            "max_s": round(lo * rng.uniform(1.0, 12.0), 2)}


# ---------------------------------------------------------------- Opus files from a seed

_sources = {}
_REV8 = bytes(int("{:08b}".format(i)[::-1], 2) for i in range(256))


def _ogg_crc(page):
    """Ogg's checksum (polynomial 0x04c11db7, not reflected, initial value 0) by the reflected crc32."""
    r = zlib.crc32(page.translate(_REV8), 0xFFFFFFFF) ^ 0xFFFFFFFF
    return int("{:032b}".format(r)[::-1], 2)


def _samples48(pkt):
    """Samples at 48 kHz of one packet from its TOC byte (RFC 6716 section 3.1)."""
    cfg, code = pkt[0] >> 3, pkt[0] & 3
    q = (40, 80, 160, 240)[cfg & 3] if cfg < 12 else (40, 80)[cfg & 1] if cfg < 16 else (10, 20, 40, 80)[cfg & 3]
    return q * 12 * (1 if code == 0 else 2 if code < 3 else pkt[1] & 63)


def _source(name):
    """(packets, samples of each, start sample of each) of one encoded stream."""
    if name not in _sources:
        with open(os.path.join(GOLD, name + ".opus"), "rb") as f:
            data = f.read()
        packets, part, at = [], b"", 0
        while at < len(data):
            nseg = data[at + 26]
            lacing = data[at + 27:at + 27 + nseg]
            at += 27 + nseg
            for v in lacing:
                part += data[at:at + v]
                at += v
                if v < 255:
                    packets.append(part)
                    part = b""
        packets = packets[2:]
        n = [_samples48(p) for p in packets]
        _sources[name] = (packets, n, np.concatenate([[0], np.cumsum(n)]))
    return _sources[name]


def _packets(rng, content, seconds):
    """Packets of a file of at least `seconds` (plus pre-skip), spliced from runs of 0.5-3 s."""
    names = CONTENT[content][0]
    need, got, out, lens = int(round(seconds * 48000)) + 312, 0, [], []
    while got < need:
        p, n, start = _source(names[int(rng.integers(len(names)))])
        a = int(rng.integers(len(p)))
        b = int(np.searchsorted(start, start[a] + int(rng.uniform(0.5, 3.0) * 48000)))
        b = max(a + 1, min(b, len(p)))
        b = min(b, max(a + 1, int(np.searchsorted(start, start[a] + need - got))))   # no packets past the end
        out += p[a:b]
        lens += n[a:b]
        got += int(start[b] - start[a])
    return out, lens


def _page(serial, seq, granule, flags, lacing, body):
    head = b"OggS" + struct.pack("<BBqIII", 0, flags, granule, serial, seq, 0) + bytes([len(lacing)]) + lacing
    page = head + body
    return page[:22] + struct.pack("<I", _ogg_crc(page)) + page[26:]


def _ogg(packets, lens, channels, n_play):
    """Ogg Opus file (RFC 7845): pre-skip 312, end trim by the last page's granule."""
    head = b"OpusHead" + struct.pack("<BBHIhB", 1, channels, 312, 48000, 0, 0)
    tags = b"OpusTags" + struct.pack("<I", 4) + b"perf" + struct.pack("<I", 0)
    out = [_page(7, 0, 0, 2, bytes([len(head)]), head), _page(7, 1, 0, 0, bytes([len(tags)]), tags)]
    seq, cum, i = 2, 0, 0
    while i < len(packets):
        lacing, j = b"", i
        while j < len(packets) and j < i + 50:
            k = len(packets[j])
            if len(lacing) + k // 255 + 1 > 255:
                break
            lacing += b"\xff" * (k // 255) + bytes([k % 255])
            j += 1
        cum += sum(lens[i:j])
        last = j >= len(packets)
        out.append(_page(7, seq, min(cum, 312 + n_play) if last else cum, 4 if last else 0, lacing,
                         b"".join(packets[i:j])))
        seq, i = seq + 1, j
    return b"".join(out)


def _seconds(case):
    """Lengths of the case's files: log-uniform quantiles."""
    n, a, b = case["files"], case["min_s"], case["max_s"]
    return [a * (b / a) ** ((i + 0.5) / n) for i in range(n)]


def _kind(case, i):
    return ("mixed", "stereo")[i % 2] if case["content"] == "both" else case["content"]


def _files(case, seed):
    rng = np.random.default_rng(seed)
    made = []
    for i, s in enumerate(_seconds(case)):
        p, n = _packets(rng, _kind(case, i), s)
        made.append(_ogg(p, n, CONTENT[_kind(case, i)][1], int(round(s * 48000))))
    return [made[i] for i in np.random.default_rng(len(made)).permutation(len(made))]


# ---------------------------------------------------------------- device-resident batches

def _batch(case, seed):
    """cuopus_batch of whole streams, one chain each, and the tensors behind it."""
    rng = np.random.default_rng(seed)
    packets, npk, chans, keep = [], [], [], []
    loss = case.get("loss", 0.0)
    for i, s in enumerate(_seconds(case)):
        p, n = _packets(rng, _kind(case, i), s)
        if loss:
            gone = rng.random(len(p)) < loss
            n = [5760 if g else v for g, v in zip(gone, n)]   # a lost packet is concealed for 5760 samples
            p = [b"" if g else v for g, v in zip(gone, p)]
        packets += p
        npk.append(len(p))
        chans.append(CONTENT[_kind(case, i)][1])
        keep.append(min(int(round(s * 48000)), sum(n) - 312))
    npk, chans, keep = (np.asarray(v, np.int64) for v in (npk, chans, keep))
    lens = np.fromiter(map(len, packets), np.int64, len(packets))
    size = keep * chans
    on_gpu = lambda a, t: torch.from_numpy(np.ascontiguousarray(np.asarray(a).astype(t))).cuda()  # noqa: E731
    ends = lambda v: np.concatenate([[0], np.cumsum(v)[:-1]])  # noqa: E731
    t = dict(data=on_gpu(np.frombuffer(b"".join(packets) + bytes(16), np.uint8), np.uint8), off=on_gpu(ends(lens), np.uint64),
             len=on_gpu(lens, np.uint32), first=on_gpu(ends(npk), np.uint32), npkts=on_gpu(npk, np.uint32),
             channels=on_gpu(chans, np.uint8), trim=on_gpu(np.full(len(npk), 312), np.uint64),
             keep=on_gpu(keep, np.uint64), out_off=on_gpu(ends(size), np.uint64),
             out=torch.zeros(int(size.sum()), dtype=torch.int16, device="cuda"),
             res=torch.zeros((len(npk), 4), dtype=torch.int32, device="cuda"))
    order = np.ascontiguousarray(costmodel.packet_order(npk, chans).astype(np.uint32))
    b = cn.Batch(**{k: v.data_ptr() for k, v in t.items()})
    b.nchains, b.width, b.schedule, b.block, b.graph, b.fec = len(npk), 32, 1, 64, 0, case.get("fec", 0)
    b.order = order.ctypes.data
    return dict(batch=b, tensors=t, order=order)


def _mlp_params(seed):
    """Weights of the cost model's network (16 -> 64 -> 64 -> 1), He-scaled."""
    rng = np.random.default_rng(seed + 1)
    parts = [rng.standard_normal((16, 64)) * math.sqrt(2 / 16), rng.standard_normal(64) * 0.1,
             rng.standard_normal((64, 64)) * math.sqrt(2 / 64), rng.standard_normal(64) * 0.1,
             rng.standard_normal(64) * math.sqrt(2 / 64), rng.standard_normal(1) * 0.1]
    return np.concatenate([p.reshape(-1) for p in parts]).astype(np.float32)


_server = None   # a serving program keeps one server for its lifetime


def _the_server():
    global _server
    if _server is None:
        _server = serving.Server(budget_bytes=4 << 30)
    return _server


def _pcm(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = case["samples"]
    x = torch.randn(n, generator=g, device="cuda") * 6000.0
    return x.clamp_(-32768, 32767).to(torch.int16)


def prepare(case, seed):
    call = case["call"]
    if call == "resample":
        n = (case["samples"] - 48) // 3
        return dict(call=call, x=_pcm(case, seed), y=torch.empty(n, dtype=torch.float32, device="cuda"), n=n)
    if call in ("batch", "order"):
        state = dict(_batch(case, seed), call=call)
        if call == "order":
            state["model"] = costmodel.CostModel()
            state["model"].load(dict(params=_mlp_params(seed), mu=0.0, sigma=1.0))
        return state
    files = _files(case, seed)
    if call == "serve":
        _the_server()
    return dict(call=call, files=files)


def run(state):
    call = state["call"]
    if call == "tensor":
        return cn.decode_ogg_to_cuda_tensor(state["files"][0])
    if call == "multi":
        return cn.decode_ogg_multi(state["files"])
    if call == "channels":
        return [t for t, _ in cn.decode_ogg_to_f16k_channels(state["files"])]
    if call == "int16":
        return [t for t, _ in cn.decode_ogg_to_int16(state["files"])]
    if call == "batch":
        cn.decode_batch(state["batch"], torch.cuda.current_stream().cuda_stream)
        # samples, per chain {stop, samples, final range}; the fourth column is the measured time
        return state["tensors"]["out"], state["tensors"]["res"][:, :3]
    if call == "serve":
        srv = _the_server()
        ids = [srv.submit(f) for f in state["files"]]
        return [srv.wait(i)[0] for i in ids]
    if call == "resample":
        x, y = state["x"], state["y"]
        rc = cn.lib().cuopus_resample48to16(x.data_ptr(), x.numel(), state["n"], y.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream, None, 0)
        if rc:
            raise RuntimeError("cuopus_resample48to16: %d" % rc)
        return y
    x = costmodel.chain_features(state["batch"])
    return x, state["model"].predict_raw(x)


def work(case):
    """Packet bytes read and samples written (float32 at 16 kHz or int16 at 48 kHz); the decoder's
    operations are serial integer code of no stated count, so flops are the resampler's and the network's."""
    call = case["call"]
    if call == "resample":
        n = (case["samples"] - 48) // 3
        return {"bytes": 2 * case["samples"] + 4 * n, "flops": 2 * 49 * n}
    packed = played = 0.0
    for i, s in enumerate(_seconds(case)):
        _, ch, rate = CONTENT[_kind(case, i)]
        packed += s * rate
        played += s * ch
    if call == "order":   # each packet's TOC byte, offset and length; the features and the network
        return {"bytes": 13 * 60.0 * sum(_seconds(case)) + 68 * case["files"],
                "flops": 2 * (16 * 64 + 64 * 64 + 64) * case["files"]}
    if call in F32_CALLS:
        return {"bytes": packed + played * 64000, "flops": played * 16000 * 98}
    return {"bytes": packed + played * 96000, "flops": 0}


# ---------------------------------------------------------------- 64-bit values

def _taps():
    """49-tap Kaiser-windowed sinc (beta 8.6, cutoff 1/3, unity gain at 0 Hz), in 64 bits."""
    m = np.arange(49) - 24.0
    h = np.sinc(m / 3.0) / 3.0 * np.kaiser(49, 8.6)
    return h / h.sum()


def _mlp_exact(params, x):
    w = np.asarray(params, np.float64)
    at = 0
    parts = []
    for n in (16 * 64, 64, 64 * 64, 64, 64, 1):
        parts.append(w[at:at + n])
        at += n
    h = np.maximum(x @ parts[0].reshape(16, 64) + parts[1], 0)
    h = np.maximum(h @ parts[2].reshape(64, 64) + parts[3], 0)
    return h @ parts[4] + parts[5][0]


def _features_exact(case, seed):
    """The cost model's 16 chain features in 64 bits, from the packets' TOC bytes."""
    rng = np.random.default_rng(seed)
    rows = []
    for i, s in enumerate(_seconds(case)):
        p, n = _packets(rng, _kind(case, i), s)
        toc = np.array([q[0] for q in p])
        cfg, samples = toc >> 3, np.array(n, np.float64)
        q = np.where(cfg < 12, np.array([40, 80, 160, 240])[cfg & 3],
                     np.where(cfg < 16, np.where(cfg & 1, 80, 40), 10 << (cfg & 3)))
        nf = samples / (12 * q)
        mode = np.where(cfg < 12, 0, np.where(cfg < 16, 1, 2))
        wide = np.array([0, 2, 3, 4])[np.clip((cfg - 16) >> 2, 0, 3)]
        bw = np.where(cfg < 12, cfg >> 2, np.where(cfg < 14, 3, np.where(cfg < 16, 4, wide)))
        frames, total, secs = nf.sum(), float(sum(map(len, p))), samples.sum() / 48000
        rows.append([math.log1p(len(p)), math.log1p(total), math.log1p(frames), math.log1p(secs),
                     CONTENT[_kind(case, i)][1] - 1.0] + [nf[mode == k].sum() / frames for k in range(3)] +
                    [nf[q == k].sum() / frames for k in (10, 20, 40, 80)] + [nf[q > 80].sum() / frames] +
                    [(nf * bw).sum() / frames / 4, ((toc >> 2) & 1).mean(), math.log1p(total / secs)])
    return np.array(rows)


def exact(case, seed):
    """The resampler's and the cost model's values in 64 bits.  Decoded files have none: without this
    repository's code there is no Opus decoder, and its int16 samples are whole numbers."""
    if case["call"] == "resample":
        n, taps = (case["samples"] - 48) // 3, torch.from_numpy(_taps())
        x = torch.nn.functional.pad(_pcm(case, seed), (24, 64))
        y = torch.zeros(n, dtype=torch.float64, device=x.device)
        for k in range(49):   # output i is centred on input 3 i
            y += float(taps[k]) / 32768.0 * x[k:k + 3 * n:3][:n]
        return y
    if case["call"] == "order":
        x = _features_exact(case, seed)
        return x, _mlp_exact(_mlp_params(seed), x)
    return None
