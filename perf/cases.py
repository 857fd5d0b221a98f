"""Workloads of the PUSCH receiver equalization path, as its users call it.

Each case is one call (or one slot loop's turn) of a public entry point on
seeded synthetic slots.  Shapes are those of the benchmark configurations and
of the tests, or generic ones; ``draw`` gives more of the same ranges.

Slots: H[sc][ant][layer] has E|h|^2 = 1/nAnt, transmitted symbols are uniform
square QAM of unit energy, Y[sc][sym][ant] = H x + CN(0, sigma2) with
sigma2 = 10^(-SNR/10).
"""
from __future__ import annotations

import importlib
import math
import random
import weakref

import numpy as np
import torch

DEV = "cuda"
QAM_BITS = {4: 1, 16: 2, 64: 3, 256: 4}      # QAM order -> bits per real dimension
PRBS, ANTS, LAYERS = (24, 51, 106, 132, 273), (16, 32, 64), (2, 4, 8)
MOST_BYTES = 1.25e9                          # inputs and outputs of a drawn case


def _lib():
    return importlib.import_module("aerial-mimo-tc-optimization_b200")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _eq(slots, prb, ant, lay, sym, qam, snr, chan="iid", prec="fp16", half=False, **more):
    return dict(kind="eq", slots=slots, prb=prb, ant=ant, lay=lay, sym=sym, qam=qam, snr=snr, chan=chan, prec=prec,
                half=half, **more)


def listed():
    return [
        # one 20 MHz cell's slot: the smallest call a base station makes, where latency counts
        _eq(1, 24, 32, 4, 11, 16, 20.0, name="eq 1 slot 24x32x4"),
        # one slot of the 100 MHz massive-MIMO cell, the reference's workload, alone: a cell served by itself
        _eq(1, 132, 64, 8, 11, 256, 25.0, "prb", name="eq 1 slot 132x64x8"),
        # 64 such slots in one launch: a baseband pool at full load
        _eq(64, 132, 64, 8, 11, 256, 25.0, "prb", name="eq 64 slots 132x64x8"),
        # full-band cell with many layers on a correlated channel, where split-precision operands are needed
        _eq(12, 273, 128, 16, 11, 256, 30.0, "corr", "bf16x3", name="eq 12 slots 273x128x16 bf16x3"),
        # half-precision storage of samples, channel and LLRs: a front end that delivers complex half
        _eq(64, 132, 64, 8, 11, 256, 25.0, "prb", half=True, name="eq 64 slots 132x64x8 half"),
        # 16 cells of different widths, antennas, layers and modulations, one replayed graph: a site's slot
        dict(kind="mix", name="eq 16 uneven cells graph", cells=16, ragged=False, shapes=42, prec="fp16", graph=True),
        # cells whose layers, antennas and symbols fill no tile: partly loaded cells, odd antenna panels
        dict(kind="mix", name="eq 12 ragged cells", cells=12, ragged=True, shapes=7, prec="fp16", graph=False),
        # the FP32 chain stage by stage: users who need the reference's results bit for bit
        dict(kind="plain", name="plain chain 4 slots 132x64x8", slots=4, prb=132, ant=64, lay=8, sym=11, qam=256,
             snr=25.0),
        # the reference's own pipeline of kernels: Gram, tensor-core coef_apply, demapper (coefficients in hand)
        dict(kind="stages", name="stages 8 slots 132x64x8", slots=8, prb=132, ant=64, lay=8, sym=14, qam=256,
             snr=25.0),
        # SRS channel estimation of 40 cells, 4 symbols each
        dict(kind="srs", name="srs 10560 blocks", blocks=10560, ant=64, taps=24, outs=24, ports=4, occ=4, half=True),
        # DMRS interpolation of 40 full-band cells into the channel the equalizer reads
        dict(kind="chest", name="chest 2720 blocks", blocks=2720, ant=64, taps=96, outs=96, ports=4, occ=4,
             half=False),
        # the serving loop: 40 cells hand in one slot each, two of them after an SRS update of their channel
        dict(kind="serve", name="serve 40 cells", cells=40, updates=2, shapes=42),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _fit(case, key, low=1):
    """Halves case[key] until the case's bytes are those of the largest listed one or fewer."""
    while case[key] > low and work(case)["bytes"] > MOST_BYTES:
        case[key] = max(low, case[key] // 2)
    return case


def draw(rng):
    kind = rng.choice(("eq", "eq", "eq", "mix", "ragged", "plain", "stages", "srs", "chest", "serve"))
    qam, snr = rng.choice((4, 16, 64, 256)), round(rng.uniform(10.0, 30.0), 1)
    if kind == "eq":
        half = rng.random() < 0.25
        ant = rng.choice((16, 32, 64, 128) if half else (16, 24, 32, 48, 64, 64, 96, 128))
        lay = rng.choice([v for v in ((2, 4, 8, 16) if half else (1, 2, 3, 4, 4, 6, 8, 8, 12, 16)) if 2 * v <= ant])
        return _fit(_eq(_log_int(rng, 1, 64), _log_int(rng, 5, 273), ant, lay, rng.randint(7, 14), qam, snr,
                        rng.choice(("iid", "prb", "corr")),
                        "fp16" if half else rng.choice(("fp16", "fp16", "bf16x3", "fp16x3")), half), "slots")
    if kind in ("mix", "ragged"):
        return dict(kind="mix", cells=rng.randint(4, 48), ragged=kind == "ragged", shapes=rng.randint(100, 1 << 20),
                    prec=rng.choice(("fp16", "fp16", "bf16x3")), graph=rng.random() < 0.5)
    if kind in ("plain", "stages"):
        ant = rng.choice((16, 24, 32, 48, 64, 128))
        lay = rng.choice([v for v in (1, 2, 3, 4, 6, 8, 8, 16) if 2 * v <= ant])
        return dict(kind=kind, slots=rng.randint(1, 4), prb=_log_int(rng, 5, 273), ant=ant, lay=lay,
                    sym=rng.randint(7, 14), qam=qam, snr=snr)
    if kind in ("srs", "chest"):
        taps = rng.choice((12, 18, 24, 24, 48)) if kind == "srs" else rng.choice((12, 24, 48, 72, 96))
        return _fit(dict(kind=kind, blocks=_log_int(rng, 40, 10560 if kind == "srs" else 2720),
                         ant=rng.choice((16, 32, 48, 64)), taps=taps,
                         outs=taps if kind == "srs" else taps * rng.choice((1, 1, 2)), ports=rng.choice((2, 4, 4, 8)),
                         occ=rng.choice((2, 4)), half=kind == "srs" or rng.random() < 0.4), "blocks")
    return dict(kind="serve", cells=rng.randint(4, 40), updates=rng.randint(0, 3), shapes=rng.randint(100, 1 << 20))


def _mix_shapes(case):
    """(prb, ant, lay, sym, qam, snr) of every cell of a mixed batch."""
    r, out = random.Random(case["shapes"]), []
    for _ in range(case["cells"]):
        if case.get("ragged"):
            ant = r.choice((8, 12, 16, 20, 24, 32, 40, 48, 64, 100))
            lay = r.randint(1, min(12, ant // 2))
            out.append((r.randint(1, 106), ant, lay, r.randint(5, 14), r.choice((4, 16, 64, 256)), r.uniform(10, 30)))
        else:
            out.append((r.choice(PRBS), r.choice(ANTS), r.choice(LAYERS), 11, r.choice((4, 16, 64, 256)),
                        r.uniform(10, 30)))
    return out


def _eq_work(nsc, ant, lay, sym, qam, cs):
    """Bytes (cs per complex sample, cs/2 per LLR) and FLOPs (8 per complex multiply-add; the Gram's and the
    factor's lower triangles) of the chain over nsc subcarriers."""
    n = QAM_BITS[qam]
    by = nsc * (cs * ant * lay + cs * ant * sym + cs // 2 * lay * sym * 2 * n)
    fl = nsc * (4 * ant * lay * (lay + 1) + 8 * ant * lay * sym + 8 * lay ** 3 / 3 + 8 * lay * lay * sym)
    return by, fl


def work(case):
    k = case["kind"]
    if k == "eq":
        by, fl = _eq_work(case["slots"] * 12 * case["prb"], case["ant"], case["lay"], case["sym"], case["qam"],
                          4 if case["half"] else 8)
    elif k in ("mix", "serve"):
        w = [_eq_work(12 * p, a, l, s, q, 8) for p, a, l, s, q, _ in _mix_shapes(case)]
        by, fl = sum(x[0] for x in w), sum(x[1] for x in w)
    elif k == "plain":
        by, fl = _eq_work(case["slots"] * 12 * case["prb"], case["ant"], case["lay"], case["sym"], case["qam"], 8)
    elif k == "stages":
        a, l, s, n = case["ant"], case["lay"], case["sym"], QAM_BITS[case["qam"]]
        nsc = case["slots"] * 12 * case["prb"]
        gram, apply, demap = 8 * (a * l + l * l), 8 * (l * a + s * a + l * s), 8 * l * s + 4 * l + 4 * l * s * 2 * n
        by, fl = nsc * (gram + apply + demap), nsc * 8 * (a * l * (l + 1) / 2 + l * a * s)
    else:
        m, n = case["blocks"] * case["ant"], case["outs"] * case["ports"]
        by = 4 * m * case["taps"] + (4 if case["half"] else 8) * m * n + 4 * case["outs"] * case["taps"]
        fl = 8 * m * n * case["taps"]
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _cn(shape, var, g):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.complex64) * math.sqrt(var)


def _channel(nsc, ant, lay, chan, g):
    """i.i.d. taps; "prb": constant over 12 subcarriers plus a small perturbation; "corr": exponential
    correlation 0.7 over the antennas."""
    if chan == "prb":
        return (_cn((nsc // 12, 1, ant, lay), 1 / ant, g).expand(-1, 12, -1, -1).reshape(nsc, ant, lay)
                + _cn((nsc, ant, lay), 0.01 / ant, g))
    h = _cn((nsc, ant, lay), 1 / ant, g)
    if chan == "corr":
        i = np.arange(ant)
        r = torch.from_numpy(np.linalg.cholesky(0.7 ** np.abs(i[:, None] - i[None, :]))).to(DEV, torch.complex64)
        h = torch.matmul(r, h)
    return h


def _received(h, sym, qam, snr, g):
    """Received samples of uniform QAM symbols through h, and the noise variance."""
    nsc, _, lay = h.shape
    n = QAM_BITS[qam]
    iq = torch.randint(0, 1 << n, (2, nsc, lay, sym), generator=g, device=DEV)
    iq = (2 * iq - ((1 << n) - 1)).to(torch.float32) / math.sqrt(2 * (4 ** n - 1) / 3)
    s2 = 10.0 ** (-snr / 10)
    y = torch.matmul(h, torch.complex(iq[0], iq[1])).transpose(1, 2)
    return y + _cn(y.shape, s2, g), s2


def _slot(nsc, ant, lay, sym, qam, snr, chan, g):
    h = _channel(nsc, ant, lay, chan, g)
    y, s2 = _received(h, sym, qam, snr, g)
    return h.contiguous(), y.contiguous(), s2


def _pairs(z):
    """complex64 -> float16 (re, im) pairs."""
    return torch.view_as_real(z).to(torch.float16).contiguous()


def _srs_inputs(blocks, ant, taps, outs, ports, occ, seed):
    """Pilots, a smoothing filter (a band around the diagonal) and unit-modulus cover codes, complex half."""
    g = _gen(seed)
    at = torch.arange(outs, device=DEV)[:, None] * (taps / outs) - torch.arange(taps, device=DEV)[None, :]
    w = torch.exp(-at.square() / 8.0) * torch.exp(2j * math.pi * 0.01 * at)
    w = w / w.abs().square().sum(1, keepdim=True).sqrt()
    w = w + _cn(w.shape, 1e-4, g)
    code = torch.exp(2j * math.pi * torch.arange(ports, device=DEV)[:, None] * torch.arange(occ, device=DEV) / occ)
    return _pairs(_cn((blocks, ant, taps), 1 / ant, g)), _pairs(w), _pairs(code.to(torch.complex64))


def _filtered(srs, w, code, dt):
    """H[blk][out][ant][port] = sum_k w[out][k] code[port][k mod occ] srs[blk][ant][k] of half pairs, in dt."""
    s, w, code = (torch.view_as_complex(t.to(torch.float64)).to(dt) for t in (srs, w, code))
    blocks, ant, taps = s.shape
    t = w[:, None, :] * code[:, torch.arange(taps, device=DEV) % code.shape[1]][None]       # [out][port][k]
    h = torch.matmul(s.reshape(blocks * ant, taps), t.reshape(-1, taps).T)
    return h.reshape(blocks, ant, w.shape[0], code.shape[0]).transpose(1, 2)


def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    g, k = _gen(seed), case["kind"]
    if k in ("eq", "plain", "stages"):
        h, y, s2 = _slot(case["slots"] * 12 * case["prb"], case["ant"], case["lay"], case["sym"], case["qam"],
                         case["snr"], case.get("chan", "prb"), g)
        return (_pairs(h), _pairs(y), s2) if case.get("half") else (h, y, s2)
    if k == "mix":
        return [_slot(12 * p, a, l, s, q, snr, "iid", g) for p, a, l, s, q, snr in _mix_shapes(case)]
    if k == "serve":
        out = []
        for i, (p, a, l, s, q, snr) in enumerate(_mix_shapes(case)):
            h, up = _channel(12 * p, a, l, "iid", g), None
            seen = h
            if i < case["updates"]:          # this slot goes through the channel that its SRS update estimates
                up = _srs_inputs(4 * p, a, 12, 12, l, 4, seed * 100 + i)
                seen = _srs_channel(up, torch.complex64)
            out.append((h.contiguous(), up) + tuple(_received(seen.contiguous(), s, q, snr, g)))
        return out
    return _srs_inputs(case["blocks"], case["ant"], case["taps"], case["outs"], case["ports"], case["occ"], seed)


def _srs_channel(up, dt):
    """The channel that an SRS update over 4 symbols estimates: the average of their filter outputs."""
    h = _filtered(*up, dt)
    b, k, a, p = h.shape
    return h.reshape(4, b // 4 * k, a, p).mean(0)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _coefficients(h, s2, dt):
    """Unbiased MMSE coefficients C[sc][layer][ant] and 1 / noise variance per (sc, layer)."""
    h = h.to(dt)
    hh = h.mH
    gi = torch.linalg.inv(torch.matmul(hh, h) + s2 * torch.eye(h.shape[2], device=DEV, dtype=dt))
    t = s2 * torch.diagonal(gi, dim1=1, dim2=2).real
    return torch.matmul(gi, hh) / (1 - t)[..., None], (1 - t) / t


def prepare(case, seed):
    aeq, k = _lib(), case["kind"]
    st = dict(case=case, aeq=aeq)
    ins = _inputs(case, seed)
    if k in ("eq", "plain"):
        h, y, s2 = ins
        n, half = QAM_BITS[case["qam"]], case.get("half", False)
        nsc, fmt = 12 * case["prb"], aeq.FMT_CF16 if half else aeq.FMT_CF32
        llr = torch.empty((case["slots"], nsc, case["lay"], case["sym"], 2 * n), device=DEV,
                          dtype=torch.float16 if half else torch.float32)
        st.update(keep=(h, y), out=llr, cells=[
            aeq.cell_desc(h[i * nsc:(i + 1) * nsc], y[i * nsc:(i + 1) * nsc], llr[i], s2, case["prb"], case["ant"],
                          case["lay"], case["sym"], n, fmt=fmt) for i in range(case["slots"])])
        if k == "plain":
            st["ws"] = torch.empty(aeq.pusch_eq_plain_workspace(st["cells"]), device=DEV, dtype=torch.uint8)
        else:
            st["tuning"] = aeq.make_tuning(case["prec"])
    elif k == "mix":
        out, cells = [], []
        for (h, y, s2), (p, a, l, s, q, _) in zip(ins, _mix_shapes(case)):
            out.append(torch.empty((12 * p, l, s, 2 * QAM_BITS[q]), device=DEV))
            cells.append(aeq.cell_desc(h, y, out[-1], s2, p, a, l, s, QAM_BITS[q]))
        st.update(keep=ins, out=out, cells=cells, tuning=aeq.make_tuning(case["prec"]))
        if case["graph"]:
            st["graph"] = aeq.FusedGraph(cells, st["tuning"])
            weakref.finalize(st["graph"], _destroy_graph, aeq, st["graph"]._h)
    elif k == "stages":
        h, y, s2 = ins
        nsc, l, s = h.shape[0], case["lay"], case["sym"]
        c, ni = _coefficients(h, s2, torch.complex64)
        st.update(h=h, y=y, s2=s2, c=c.contiguous(), ni=ni.contiguous(),
                  gram=torch.empty((nsc, l, l), device=DEV, dtype=torch.complex64),
                  yeq=torch.empty((nsc, l, s), device=DEV, dtype=torch.complex64),
                  llr=torch.empty((nsc, l, s, 2 * QAM_BITS[case["qam"]]), device=DEV))
    elif k in ("srs", "chest"):
        n, b = case["outs"], case["blocks"]
        shape = (b, case["ant"], n, case["ports"]) if k == "srs" else (b, n, case["ant"], case["ports"])
        st.update(ins=ins, out=torch.empty(shape + (2,), device=DEV,
                                           dtype=torch.float16 if case["half"] else torch.float32))
    else:
        srv = aeq.Server(streams=2, batch_window_us=20.0, min_batch=2)
        weakref.finalize(srv, _destroy_server, aeq, srv._h)
        st.update(srv=srv, keep=ins, out=[], jobs=[])
        torch.cuda.current_stream().synchronize()      # the server's streams read what was made on this one
        for (h, up, y, s2), (p, a, l, s, q, _) in zip(ins, _mix_shapes(case)):
            cid = srv.add_cell(p, a, l, s, QAM_BITS[q], s2)
            srv.set_channel(cid, h, s2)
            st["out"].append(torch.empty((12 * p, l, s, 2 * QAM_BITS[q]), device=DEV))
            st["jobs"].append((cid, up, y.contiguous(), st["out"][-1]))
        torch.cuda.current_stream().synchronize()
    return st


def _destroy_graph(aeq, handle):
    torch.cuda.synchronize()
    aeq.lib().aerial_eq_graph_destroy(handle)


def _destroy_server(aeq, handle):
    aeq.lib().aerial_server_destroy(handle)


def run(st):
    aeq, case = st["aeq"], st["case"]
    k = case["kind"]
    if "graph" in st:
        st["graph"].launch()
        return st["out"]
    if k in ("eq", "mix"):
        aeq.pusch_eq_fused(st["cells"], st["tuning"])
        return st["out"]
    if k == "plain":
        aeq.pusch_eq_plain(st["cells"], st["ws"])
        return st["out"]
    if k == "stages":
        nsc, a, l, s = st["h"].shape[0], case["ant"], case["lay"], case["sym"]
        aeq.gram(st["h"], st["s2"], st["gram"], nsc, a, l)
        aeq.coef_apply_tc(st["c"], st["y"], st["yeq"], nsc, s, l, a)
        aeq.llr_f32(st["yeq"], st["ni"], st["llr"], nsc * l * s, QAM_BITS[case["qam"]], s)
        return {"gram": st["gram"], "yeq": st["yeq"], "llr": st["llr"]}
    if k == "srs":
        x, w, code = st["ins"]
        aeq.srs_filter(st["out"], x, w, code, case["ant"], case["blocks"], case["taps"], case["ports"], case["occ"])
        return st["out"]
    if k == "chest":
        x, w, code = st["ins"]
        call = aeq.chest_interp_h if case["half"] else aeq.chest_interp
        call(st["out"], x, w, code, case["ant"], case["blocks"], case["taps"], case["outs"], case["ports"],
             case["occ"])
        return st["out"]
    srv = st["srv"]
    for cid, up, y, llr in st["jobs"]:
        if up is not None:
            srv.srs_update(cid, *up, 12, 4, n_symbols=4)
        srv.submit(cid, y, llr)
    srv.drain()
    srv.poll()
    return st["out"]


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _llr64(x, ni, qam):
    """Max-log LLRs [..., 2 bits] (bit, then I / Q) of x[sc][layer][sym] with 1 / noise variance ni[sc][layer]."""
    n = QAM_BITS[qam]
    norm = math.sqrt(2 * (4 ** n - 1) / 3)
    dist = 1 / norm
    out = torch.empty(x.shape + (n, 2), device=DEV, dtype=torch.float64)
    for iq, sb in enumerate((x.real, x.imag)):
        soft, near = [], []
        for i in range(n):
            soft.append(sb)
            near.append((dist + sb.abs()).square())
            if i < n - 1:
                sb = 2 ** (n - 1 - i) / norm - sb.abs()
        last = (sb.abs() - dist).square()
        for i in range(n):
            v = (near[i] - last) * ni[..., None]
            out[..., i, iq] = torch.where(soft[i] < 0, -v, v).clamp(-65504.0, 65504.0)
    return out.reshape(x.shape + (2 * n,))


def _chain64(h, y, s2, qam):
    """LLRs of every subcarrier, some thousand at a time."""
    out = []
    step = max(12, (1 << 24) // (h.shape[1] * h.shape[2]))
    for i in range(0, h.shape[0], step):
        c, ni = _coefficients(h[i:i + step], s2, torch.complex128)
        x = torch.matmul(c, y[i:i + step].to(torch.complex128).transpose(1, 2))
        out.append(_llr64(x, ni, qam))
    return torch.cat(out)


def _f32(v):
    return float(np.float32(v))       # the noise variance as the descriptors carry it


def exact(case, seed):
    k, ins = case["kind"], _inputs(case, seed)
    if k in ("eq", "plain"):
        h, y, s2 = ins
        if case.get("half"):
            h, y = (torch.view_as_complex(t.to(torch.float32)) for t in (h, y))
        v = _chain64(h, y, _f32(s2), case["qam"])
        return v.reshape((case["slots"], -1) + v.shape[1:])
    if k == "mix":
        return [_chain64(h, y, _f32(s2), c[4]) for (h, y, s2), c in zip(ins, _mix_shapes(case))]
    if k == "serve":
        return [_chain64(h if up is None else _srs_channel(up, torch.complex128), y, _f32(s2), c[4])
                for (h, up, y, s2), c in zip(ins, _mix_shapes(case))]
    if k == "stages":
        h, y, s2 = ins
        c, ni = _coefficients(h, s2, torch.complex64)          # the inputs of the later stages
        h = h.to(torch.complex128)
        gram = torch.matmul(h.mH, h) + _f32(s2) * torch.eye(h.shape[2], device=DEV)
        x = torch.matmul(c.to(torch.complex128), y.to(torch.complex128).transpose(1, 2))
        return {"gram": gram, "yeq": x, "llr": _llr64(x, ni.to(torch.float64), case["qam"])}
    v = _filtered(*ins, torch.complex128)
    return (v.transpose(1, 2) if k == "srs" else v).contiguous()
