"""Timed cases of the smartpca framework, through its Python entry points (eig_gb300.native).

A case's "kind" says which part of the framework one pass runs:

  run      a whole smartpca job on host records: upload, filters, Gram, eigensolve, outlier
           check, SNP weights, lsqproject (gp_smartpca_run, what the command-line tool calls)
  gram     one pass over a resident panel: counts, normalisation, Gram (gp_xtx)
  pca      that pass and the eigensolve (gp_xtx, gp_eigvecs)
  project  SNP weights and lsqproject after a PCA (gp_snp_weights, gp_lsqproj)
  fast     fastmode, the block Krylov PCA (gp_fastpca)
  serve    a burst of projection requests to a server on a resident panel (gp_serve_*)
  convert  re-encoding a resident panel's records (gp_encode_records, convertf)
  ingest   upload of .bed records and the missing-data counts of the pre-filters

Genotypes are drawn on the GPU: populations drifting from common ancestral frequencies
(Nicholson's truncated-normal model, F between 0.005 and 0.05), a share of missing calls.
There are two more populations than eigenvectors asked for, so that these are axes of
structure, and none is so small that the outlier rule takes it for outliers.

Eigenvectors have no sign of their own: run() turns each (and what belongs to it) so that its
largest entry is positive, as a program does that compares two analyses.
"""
import math
import random

import numpy as np
import torch

from eig_gb300 import native

PREC = {"fp64": native.GP_PREC_FP64, "fp16": native.GP_PREC_SPLIT_FP16,
        "bf16x4": native.GP_PREC_SPLIT_BF16X4}
FORMATS = {"packed": native.GP_OUT_PACKEDANCESTRYMAP, "bed": native.GP_OUT_PACKEDPED,
           "eigenstrat": native.GP_OUT_EIGENSTRAT}


def listed():
    return [
        # a small cohort, the size of the repository's golden data: launches and host work
        dict(name="run_180x2500_fp64", kind="run", n=180, m=2500, k=10, prec="fp64", miss=0.02,
             code="packed"),
        # a genotyping study at the default (FP64) precision
        dict(name="run_1000x50000_fp64", kind="run", n=1000, m=50000, k=10, prec="fp64",
             miss=0.01, code="packed"),
        # the benchmark's workload: a biobank-sized panel at split precision
        dict(name="run_5000x600000_fp16", kind="run", n=5000, m=600000, k=20, prec="fp16",
             miss=0.02, code="packed"),
        # the Gram of a ragged panel at the default precision
        dict(name="gram_2003x120011_fp64", kind="gram", n=2003, m=120011, prec="fp64", miss=0.02,
             plo=0.05),
        # and of one with rare variants at split precision
        dict(name="gram_3001x60007_fp16", kind="gram", n=3001, m=60007, prec="fp16", miss=0.02,
             plo=0.001),
        # the dense eigensolve of a large cohort after SNP pruning
        dict(name="pca_5000x4000", kind="pca", n=5000, m=4000, k=20, prec="fp16", miss=0.01),
        # weights and projection (poplistname: a part of the samples defines the axes)
        dict(name="project_1501x80003_fp64", kind="project", n=1501, m=80003, k=10, prec="fp64",
             miss=0.05),
        dict(name="project_5000x200000_fp16", kind="project", n=5000, m=200000, k=20,
             prec="fp16", miss=0.02),
        # fastmode on a cohort where the N x N Gram is not wanted
        dict(name="fast_10007x100003", kind="fast", n=10007, m=100003, k=10, dim=20, iters=10,
             prec="fp16", miss=0.01),
        # new samples placed on a resident panel, as they arrive
        dict(name="serve_24_of_100000", kind="serve", n=1000, m=100000, k=20, requests=24,
             most=200, miss=0.3),
        # format conversion of a biobank-sized panel
        dict(name="convert_5000x100000_bed", kind="convert", n=5000, m=100000, to="bed",
             every=True, miss=0.02),
        # reading a PLINK data set in
        dict(name="ingest_5000x100000", kind="ingest", n=5000, m=100000, miss=0.02),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "gram", "gram", "pca", "project", "project", "fast", "serve",
                       "convert", "ingest"])
    miss = round(rng.uniform(0.0, 0.1), 3)
    prec = rng.choice(["fp64", "fp64", "fp16", "bf16x4"])
    if kind == "run":
        n = _log(rng, 80, 3000)
        m = _log(rng, 1000, max(2000, min(200000, int(4e11 / n / n))))
        return dict(kind=kind, n=n, m=m, k=rng.randint(2, 10), prec=prec, miss=miss,
                    code=rng.choice(["packed", "bed"]))
    if kind == "gram":
        n = _log(rng, 80, 3000)
        m = _log(rng, 1000, max(2000, min(200000, int(5e11 / n / n))))
        return dict(kind=kind, n=n, m=m, prec=prec, miss=miss, plo=rng.choice([0.05, 0.001]))
    if kind == "pca":
        return dict(kind=kind, n=_log(rng, 100, 5000), m=rng.randint(3000, 6000),
                    k=rng.randint(2, 20), prec="fp16", miss=miss)
    if kind == "project":
        n = _log(rng, 150, 4000)
        return dict(kind=kind, n=n, m=_log(rng, 2000, max(4000, min(150000, int(2.5e8 / n)))),
                    k=rng.randint(2, 20), prec=prec, miss=miss)
    if kind == "fast":
        k = rng.randint(2, 10)
        n = _log(rng, 500, 8000)
        return dict(kind=kind, n=n, m=_log(rng, 3000, min(100000, int(6e8 / n))), k=k,
                    dim=2 * k + rng.randint(0, 3), iters=rng.randint(3, 10), prec="fp16",
                    miss=miss)
    if kind == "serve":
        return dict(kind=kind, n=_log(rng, 200, 1000), m=_log(rng, 5000, 100000),
                    k=rng.randint(2, 20), requests=rng.randint(1, 24), most=_log(rng, 1, 200),
                    miss=rng.choice([0.02, 0.3, 0.6]))
    n = _log(rng, 100, 5000)
    m = _log(rng, 2000, min(100000, int(5e8 / n)))
    if kind == "convert":
        return dict(kind=kind, n=n, m=m, to=rng.choice(["packed", "bed", "eigenstrat"]),
                    every=rng.choice([True, False]), miss=miss)
    return dict(kind=kind, n=n, m=m, miss=miss)


# ---- inputs ----------------------------------------------------------------------------

def _codes(n, m, npop, miss, plo, seed, extra=0, extra_miss=0.0, chunk=1 << 26):
    """Blocks [snps, n + extra] (uint8, on the GPU) of genotype codes 0, 1, 2 and 3 (missing);
    the last `extra` samples are new ones of the same populations."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    f = 0.005 + 0.045 * torch.rand(npop, generator=g, device="cuda")
    pop = torch.arange(n, device="cuda") * npop // n
    if extra:
        pop = torch.cat([pop, torch.randint(npop, (extra,), generator=g, device="cuda")])
    rate = torch.full((n + extra,), float(miss), device="cuda")
    rate[n:] = extra_miss
    step = max(1, chunk // (n + extra))
    for s in range(0, m, step):
        c = min(step, m - s)
        if plo < 0.05:  # rare variants: frequencies spread over their logarithm
            p = plo * (0.5 / plo) ** torch.rand(c, 1, generator=g, device="cuda")
        else:
            p = plo + (1 - 2 * plo) * torch.rand(c, 1, generator=g, device="cuda")
        q = p + (f * p * (1 - p)).sqrt() * torch.randn(c, npop, generator=g, device="cuda")
        q = q.clamp_(2e-4, 1 - 2e-4)[:, pop]
        u = torch.rand(c, n + extra, generator=g, device="cuda")
        code = torch.where(u < rate, 3.0, 0.0)
        u = (u - rate) / (1 - rate)
        code += torch.where(u < 0, 0.0, (u < q * (2 - q)).float() + (u < q * q).float())
        yield code.to(torch.uint8)


def _pack(codes, bed=False):
    """Four codes a byte along the last axis: first sample in the high bits, or PLINK's order
    and codes; what fills up the last byte is missing."""
    pad = -codes.shape[1] % 4
    if pad:
        codes = torch.cat([codes, codes.new_full((codes.shape[0], pad), 3)], 1)
    if bed:
        codes = torch.tensor([3, 2, 0, 1], dtype=torch.uint8, device=codes.device)[codes.long()]
    c = codes.view(codes.shape[0], -1, 4)
    if bed:
        return c[:, :, 0] | c[:, :, 1] << 2 | c[:, :, 2] << 4 | c[:, :, 3] << 6
    return c[:, :, 0] << 6 | c[:, :, 1] << 4 | c[:, :, 2] << 2 | c[:, :, 3]


def _panel(case, seed, npop, bed=False):
    blocks = [_pack(b, bed) for b in _codes(case["n"], case["m"], npop, case["miss"],
                                            case.get("plo", 0.05), seed)]
    return torch.cat(blocks).cpu().numpy()


def _rows(case):
    """project: the samples that define the axes (four of five); otherwise all."""
    a = np.arange(case["n"], dtype=np.int32)
    return a[a % 5 != 3] if case["kind"] == "project" else a


def _npop(case):
    return case.get("k", 10) + 2


def _request_sizes(case):
    r = random.Random(case["n"] * 1000003 + case["m"])
    return [_log(r, 1, case["most"]) for _ in range(case["requests"])]


def _loaded(case, records):
    h = native.Handle(0)
    h.load_genotypes(records, case["n"])
    h.set_samples(_rows(case))
    h.set_snps(np.arange(case["m"], dtype=np.int32))
    return h


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "run":
        bed = case["code"] == "bed"
        s["records"] = _panel(case, seed, _npop(case), bed)
        s["code"] = native.GP_CODE_BED if bed else native.GP_CODE_PACKED
        s["opts"] = native.default_opts(numeigs=case["k"], precision=PREC[case["prec"]])
        s["h"] = native.Handle(0)
    elif kind in ("gram", "pca"):
        s["h"] = _loaded(case, _panel(case, seed, _npop(case)))
    elif kind == "project":
        s["h"] = h = _loaded(case, _panel(case, seed, _npop(case)))
        h.xtx(PREC[case["prec"]], want_xtx=False)
        _, s["evecs"] = h.eigvecs(case["k"])
        s["samples"] = np.arange(case["n"], dtype=np.int32)
    elif kind == "fast":
        s["h"] = _loaded(case, _panel(case, seed, _npop(case)))
        s["omega"] = np.random.RandomState(seed % (1 << 31)).standard_normal(
            (case["n"], case["dim"]))
    elif kind == "serve":
        sizes = _request_sizes(case)
        rec, new = [], []
        for b in _codes(case["n"], case["m"], _npop(case), 0.02, 0.05, seed, sum(sizes),
                        case["miss"]):
            rec.append(_pack(b[:, :case["n"]]))
            new.append(b[:, case["n"]:].T.contiguous())
        new = torch.cat(new, 1)
        s["h"] = h = _loaded(case, torch.cat(rec).cpu().numpy())
        h.xtx(native.GP_PREC_SPLIT_FP16, want_xtx=False)
        _, s["evecs"] = h.eigvecs(case["k"])
        h.snp_weights(case["k"])
        # batches launched from the host: torch shares the device and waits for all of it
        s["server"] = v = native.Server(h, case["k"], host_loop=True)
        rows = _pack(new[:, torch.from_numpy(v.snp_index).cuda().long()])
        full = torch.full((rows.shape[0], v.row_bytes), 255, dtype=torch.uint8, device="cuda")
        full[:, :rows.shape[1]] = rows
        full = full.cpu().numpy()
        at = np.cumsum([0] + sizes)
        s["requests"] = [full[a:b] for a, b in zip(at[:-1], at[1:])]
    elif kind == "convert":
        s["h"] = h = native.Handle(0)
        h.load_genotypes(_panel(case, seed, 4), case["n"])
        r = np.random.RandomState(seed % (1 << 31))
        if case["every"]:
            s["samples"], s["snps"] = None, np.arange(case["m"])
        else:  # a part of the samples in another order, a part of the SNPs
            s["samples"] = r.permutation(case["n"])[: max(1, case["n"] * 3 // 5)]
            s["snps"] = np.sort(r.permutation(case["m"])[: case["m"] * 7 // 10])
        s["flip"] = (r.rand(len(s["snps"])) < 0.05).astype(np.uint8)
    elif kind == "ingest":
        s["h"] = native.Handle(0)
        s["records"] = _panel(case, seed, 4, bed=True)
        s["use"] = (np.arange(case["n"]) % 7 != 2).astype(np.uint8)
    return s


# ---- one pass --------------------------------------------------------------------------

def _signs(evecs):
    """[k] signs that make each row's largest entry positive"""
    at = np.argmax(np.abs(evecs), axis=1)
    return np.where(evecs[np.arange(len(evecs)), at] < 0, -1.0, 1.0)


def run(s):
    case, h = s["case"], s["h"]
    kind = case["kind"]
    if kind == "run":
        r = native.smartpca_run(h, s["records"], case["n"], s["opts"], code=s["code"])
        t = _signs(r["evecs"])[:, None]
        return dict(evals=r["evals"], evecs=r["evecs"] * t, coords=r["coords"] * t,
                    xindex=r["xindex"], snp_state=r["snp_state"], ind_out=r["ind_out"])
    if kind == "gram":
        return h.xtx(PREC[case["prec"]])
    if kind == "pca":
        x = h.xtx(PREC[case["prec"]], want_xtx=False)
        evals, evecs = h.eigvecs(case["k"])
        return dict(nused=x["nused"], evals=evals, evecs=evecs * _signs(evecs)[:, None])
    if kind == "project":
        ff, fx, sc = h.snp_weights(case["k"])
        a, b, nobs, status = h.lsqproj(case["k"], s["samples"])
        t = _signs(s["evecs"])[:, None]
        return dict(ff=ff * t, fx=fx * t, scale=sc, a=a * t, b=b * t, nobs=nobs, status=status)
    if kind == "fast":
        evals, evecs = h.fastpca(case["k"], case["dim"], case["iters"], omega=s["omega"],
                                 precision=PREC[case["prec"]])
        return dict(evals=evals, evecs=evecs * _signs(evecs)[:, None])
    if kind == "serve":
        q = [s["server"].submit(c) for c in s["requests"]]
        got = [r.wait() for r in q]
        return dict(coords=np.concatenate([c for c, _ in got]) * _signs(s["evecs"]),
                    status=np.concatenate([t for _, t in got]))
    if kind == "convert":
        return h.encode_records(FORMATS[case["to"]], s["snps"], s["samples"], s["flip"],
                                nsamples=case["n"])
    h.load_genotypes(s["records"], case["n"], native.GP_CODE_BED)
    snp, ind = h.valid_counts(s["use"], None)
    return dict(snp=snp, ind=ind)


# ---- what a pass cannot do without -----------------------------------------------------

def work(case):
    n, m, k, kind = case["n"], case["m"], case.get("k", 0), case["kind"]
    rec = m * ((n + 3) // 4)
    if kind == "convert":
        out = n * m if case["to"] == "eigenstrat" else rec
        part = 1.0 if case["every"] else 0.7
        return dict(bytes=part * rec + out * (part if case["every"] else part * 0.6), flops=0)
    if kind == "ingest":
        return dict(bytes=2 * rec + 4 * (n + m), flops=0)
    if kind == "serve":
        q = sum(_request_sizes(case))
        return dict(bytes=q * m / 4 + 8 * q * k, flops=2.0 * q * m * (k * (k + 1) / 2 + 2 * k))
    if kind == "fast":
        L, it = case["dim"], case["iters"]
        return dict(bytes=rec + 8 * n * (L + k), flops=float(n) * m * L * (6 * it + 4))
    nr = len(_rows(case))
    gram = float(nr) * (nr + 1) * m
    eig = 4.0 / 3.0 * nr ** 3
    lsq = 2.0 * n * m * (k * (k + 1) / 2 + k) + 4.0 * nr * m * k
    if kind == "gram":
        return dict(bytes=rec + 8 * n * n + 29 * m, flops=gram)
    if kind == "pca":
        return dict(bytes=rec + 8 * n * (k + 1) + 29 * m, flops=gram + eig)
    if kind == "project":
        return dict(bytes=rec + 8 * k * (m + 2 * nr + 2 * n), flops=lsq)
    return dict(bytes=rec + 8 * n * (2 * k + 1) + m, flops=gram + eig + lsq)


# ---- the same in 64 bits by torch ------------------------------------------------------

def _unpack(rec, n):
    shift = torch.tensor([6, 4, 2, 0], dtype=torch.uint8, device=rec.device)
    return ((rec[:, :, None] >> shift) & 3).view(rec.shape[0], -1)[:, :n]


class _Pass:
    """Counts, normalisation and blocks of values of one pass (every SNP, the given rows)."""

    def __init__(self, records, n, rows, least=1):
        self.rec, self.n = torch.from_numpy(records).cuda(), n
        self.rows = torch.from_numpy(rows).cuda().long()
        self.step = max(1, (1 << 26) // n)
        m = len(records)
        self.n0, self.miss = (torch.zeros(m, dtype=torch.float64, device="cuda") for _ in "01")
        for s, c in self.blocks():
            c = c[:, self.rows]
            self.n0[s] = torch.where(c == 3, 0, c).sum(1).double()
            self.miss[s] = (c == 3).sum(1).double()
        seen = len(rows) - self.miss
        self.n1 = 2 * seen - self.n0
        self.mean = self.n0 / seen
        p = self.mean / 2
        self.fancy = torch.where(p * (1 - p) > 0, 1 / (p * (1 - p)).sqrt(), 1.0)
        self.kept = torch.minimum(self.n0, self.n1) >= max(least, 1)

    def blocks(self):
        for a in range(0, len(self.rec), self.step):
            s = slice(a, min(a + self.step, len(self.rec)))
            yield s, _unpack(self.rec[s], self.n)

    def values(self, s, c):
        """normalised genotypes of the block: 0 where missing or the SNP is left out"""
        v = (c.double() - self.mean[s, None]) * self.fancy[s, None]
        return torch.where((c == 3) | ~self.kept[s, None], 0.0, v)

    def gram(self):
        k = len(self.rows)
        x = torch.zeros(k, k, dtype=torch.float64, device="cuda")
        for s, c in self.blocks():
            v = self.values(s, c[:, self.rows])
            x.addmm_(v.T, v)
        return x

    def eig(self, k):
        x = self.gram()
        x /= x.diagonal().sum() / (len(x) - 1)
        w, v = torch.linalg.eigh(x)
        v = v.flip(1)[:, :k].T.contiguous()
        t = torch.from_numpy(_signs(v.cpu().numpy())).cuda()
        return w.flip(0), v * t[:, None]

    def weights(self, evecs):
        ff = torch.zeros(len(evecs), len(self.rec), dtype=torch.float64, device="cuda")
        for s, c in self.blocks():
            ff[:, s] = 10 * evecs @ self.values(s, c[:, self.rows]).T
        fx = torch.zeros_like(evecs)
        for s, c in self.blocks():
            fx += ff[:, s] @ self.values(s, c[:, self.rows])
        return ff, fx, 1 / fx.square().sum(1).sqrt()

    def project(self, E, codes):
        """least squares of each sample's seen genotypes on E: (coefficients, right sides, seen)
        from blocks of (slice, codes [snps, samples])"""
        k = len(E)
        i, j = torch.triu_indices(k, k, device="cuda")
        co = rr = seen = 0
        for s, c in codes:
            e = E[:, s] * self.kept[s]
            o = ((c != 3) & self.kept[s, None]).double()
            co = co + (e[i] * e[j]) @ o
            rr = rr + e @ self.values(s, c)
            seen = seen + o.sum(0)
        A = torch.zeros(co.shape[1], k, k, dtype=torch.float64, device="cuda")
        A[:, i, j] = co.T
        A[:, j, i] = co.T
        return torch.linalg.solve(A, rr.T).T, rr, seen


def _host(**d):
    return {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in d.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("convert", "ingest"):
        return None
    if kind != "fast" and case["n"] ** 2 * float(case["m"]) > 6e12:
        return None
    k = case.get("k", 0)
    if kind == "serve":
        sizes = _request_sizes(case)
        blocks = list(_codes(case["n"], case["m"], _npop(case), 0.02, 0.05, seed, sum(sizes),
                             case["miss"]))
        p = _Pass(torch.cat([_pack(b[:, :case["n"]]) for b in blocks]).cpu().numpy(), case["n"],
                  _rows(case))
        ff, _, sc = p.weights(p.eig(k)[1])
        new = torch.cat([b[:, case["n"]:] for b in blocks])
        cut = max(1, (1 << 26) // (new.shape[1] + k * k))
        a, _, _ = p.project(ff * sc[:, None], ((slice(i, i + cut), new[i:i + cut])
                                               for i in range(0, len(new), cut)))
        return _host(coords=a.T, status=None)
    rec = _panel(case, seed, _npop(case))
    p = _Pass(rec, case["n"], _rows(case))
    if kind == "gram":
        x = p.gram()
        return _host(n0=None, n1=None, nmiss=None, killed=None, xmean=p.mean * p.fancy,
                     xfancy=p.fancy, XTX=x, trace=float(x.diagonal().sum()), nused=None)
    if kind == "fast":
        vals = [p.values(s, c) for s, c in p.blocks()]  # the block Krylov space of X'X
        m = case["m"]

        def down(g):
            return torch.cat([v @ g for v in vals]) / math.sqrt(2.0)

        def up(q):
            at = np.cumsum([0] + [len(v) for v in vals])
            return sum(v.T @ q[a:b] for v, a, b in zip(vals, at[:-1], at[1:])) / math.sqrt(2.0)

        g = torch.from_numpy(np.random.RandomState(seed % (1 << 31)).standard_normal(
            (case["n"], case["dim"]))).cuda()
        basis = None
        for _ in range(case["iters"] + 1):
            q = down(g)
            g = up(q) / m
            for _ in range(2):
                if basis is not None:
                    q = q - basis @ (basis.T @ q)
                q = torch.linalg.qr(q)[0]
            basis = q if basis is None else torch.cat([basis, q], 1)
        b = up(basis)
        w, z = torch.linalg.eigh(b.T @ b)
        evecs = (b @ z.flip(1)[:, :k] / w.flip(0)[:k].sqrt()).T
        t = torch.from_numpy(_signs(evecs.cpu().numpy())).cuda()
        return _host(evals=w.flip(0)[:k] / m, evecs=evecs * t[:, None])
    evals, evecs = p.eig(k)
    if kind == "pca":
        return _host(nused=None, evals=evals, evecs=evecs)
    ff, fx, sc = p.weights(evecs)
    a, b, _ = p.project(ff * sc[:, None], p.blocks())
    if kind == "project":
        return _host(ff=ff, fx=fx, scale=sc, a=a, b=b, nobs=None, status=None)
    a = a * ((a * b).sum(1) / a.square().sum(1))[:, None]
    return _host(evals=evals, evecs=evecs, coords=a, xindex=None, snp_state=None, ind_out=None)
