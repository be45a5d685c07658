"""The work that programs built on ngia2_gb300 have it do, as timed cases.

Seven kinds of program, each through the package's public entry points:

  cluster  a database resident on the device: sketch, bucket, candidates,
           alignment and edges copied to the host (Context.group_align +
           ngia_ctx_edges), what `-m clustering` does between reading its file
           and Leiden
  host     the same from page-locked host buffers to host edges in one call
           (Context.run_host), a loop over databases with one context
  fast     fast mode: sketch + bucket, then greedy clustering
           (Context.sketch_bucket + Context.fast_cluster), `-m fast`
  pairs    batched alignment of a caller's candidate pairs
           (Context.align_pairs_device)
  raw      the four device-pointer entry points that stand in for the
           reference's own stages (sketch, bucket, align_pairs, emit_edges)
  serve    requests of query sequences against a resident database
           (Server.submit + Server.wait)
  stream   records in host memory streamed through a device budget
           (ngia_stream_graph)

Edges land in a buffer that the program keeps (zeros beyond their count), so
an output's shape depends on its case alone.

Sequences are families from the generators of ngia2_gb300.synth (same length
distributions, substitution and indel rates), drawn on the GPU.  Every output
is a whole number (scores, indices, cluster ids, signatures; edges are
returned as their 32-bit words, the weight's bit pattern included), so outputs
are equal or wrong and no 64-bit value is needed.
"""
import ctypes
import math

import numpy as np
import torch

import ngia2_gb300 as ng

DEV = "cuda"
AMINO = b"ACDEFGHIKLMNPQRSTVWY"
AMINO_FREQ = [8.25, 1.37, 5.45, 6.75, 3.86, 7.07, 2.27, 5.96, 5.84, 9.66,
              2.42, 4.06, 4.70, 3.93, 5.53, 6.56, 5.34, 6.87, 1.08, 2.92]
NUCLEO = b"ACGT"
NUCLEO_FREQ = [0.275, 0.225, 0.225, 0.275]  # GC = 0.45
MEAN_LEN = {"protein": 340, "protein_close": 340, "dna": 1600, "dna_n": 1600, "mixed": 1000}


def listed():
    return [
        # a few hundred proteins, an interactive call: launches and latency
        dict(name="cluster_protein_600", kind="cluster", seqs="protein", n=600, families=60,
             identity=50, bands=64),
        # the small-protein configuration
        dict(name="cluster_protein_20k", kind="cluster", seqs="protein", n=20_000,
             families=2_000, identity=90, bands=64),
        # a large, odd-sized protein set at the lowest usual identity: wide bands
        dict(name="cluster_protein_1m", kind="cluster", seqs="protein", n=1_000_003,
             families=100_000, identity=50, bands=64),
        # the nucleotide configuration, database resident
        dict(name="cluster_dna_200k", kind="cluster", seqs="dna", n=200_000, families=20_000,
             identity=95, bands=64),
        # reads with ambiguous letters: five codes, no 8-mer tables
        dict(name="cluster_dna_n_25k", kind="cluster", seqs="dna_n", n=25_013, families=2_501,
             identity=85, bands=64),
        # the nucleotide configuration from host buffers to host edges
        dict(name="host_dna_200k", kind="host", seqs="dna", n=200_000, families=20_000,
             identity=95, bands=64),
        # fast mode on a protein set of that size with many close relatives, the
        # redundancy that greedy clustering is run to remove
        dict(name="fast_protein_20k", kind="fast", seqs="protein_close", n=20_000,
             families=2_000, identity=90, bands=64),
        # the batched-alignment configuration: 2,000,000 heavy-tailed pairs
        dict(name="pairs_2m", kind="pairs", seqs="mixed", pairs=2_000_000, identity=90),
        # the drop-in entry points on one small-protein set, four bands' jobs
        dict(name="raw_protein_20k", kind="raw", seqs="protein", n=20_000, families=2_000,
             identity=90, job_bands=4),
        # one small request to a server: the latency a single user sees
        dict(name="serve_small", kind="serve", seqs="protein_close", n=100_000, families=5_000,
             requests=1, least=5, most=5, identity=90),
        # a burst of requests of log-uniform sizes, most queries with close relatives
        dict(name="serve_mix", kind="serve", seqs="protein_close", n=100_000, families=5_000,
             requests=24, least=1, most=20_000, identity=90),
        # a database in host memory through a small device budget, three bands
        dict(name="stream_400k", kind="stream", seqs="protein", n=400_009, families=33_334,
             identity=50, bands=3, chunk_mib=64),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cluster", "cluster", "cluster", "host", "fast", "pairs", "raw", "serve",
                       "stream"])
    if kind == "pairs":
        return dict(kind=kind, seqs="mixed", pairs=_log_uniform(rng, 1_000, 1_900_000),
                    identity=rng.randint(80, 95))
    if kind == "serve":
        n, seqs = _log_uniform(rng, 10_000, 100_000), rng.choice(["protein", "protein_close"])
        return dict(kind=kind, seqs=seqs, n=n, families=n // 20, requests=rng.randint(1, 24),
                    least=1, most=_log_uniform(rng, 50, 20_000),
                    identity=rng.choice([50, 60, 70] if seqs == "protein" else [80, 90, 95]))
    if kind == "stream":
        n = _log_uniform(rng, 100_000, 400_000)
        return dict(kind=kind, seqs="protein", n=n, families=n // 12,
                    identity=rng.choice([50, 70, 90]), bands=rng.choice([1, 2, 3]),
                    chunk_mib=rng.choice([64, 128, 256]))
    most = {"cluster": {"protein": 1_000_000, "protein_close": 1_000_000, "dna": 200_000,
                        "dna_n": 25_000},
            "host": {"protein": 400_000, "dna": 200_000},
            "fast": {"protein": 20_000, "protein_close": 20_000, "dna": 10_000, "dna_n": 5_000},
            "raw": {"protein": 20_000, "dna": 5_000}}[kind]
    seqs = rng.choice(sorted(most))
    most = most[seqs]
    n = _log_uniform(rng, 1_000 if kind == "fast" else 200, most)
    case = dict(kind=kind, seqs=seqs, n=n, families=max(1, n // 10),
                identity=rng.randint(80, 98) if "dna" in seqs else rng.randint(50, 95))
    if kind == "fast" and seqs != "protein_close":  # identities that families still reach
        case["identity"] = rng.randint(80, 92) if "dna" in seqs else rng.randint(50, 70)
    if kind == "raw":
        case["job_bands"] = rng.randint(1, 4)
    else:
        case["bands"] = rng.choice([64, 64, rng.randint(1, 63)])
    return case


# ---- sequences --------------------------------------------------------------------------
def _draw(g, alphabet, freqs, k):
    cdf = torch.cumsum(torch.tensor(freqs, dtype=torch.float64), 0)
    cdf = (cdf / cdf[-1]).to(torch.float32)[:-1].to(DEV)
    letters = torch.tensor(list(alphabet), dtype=torch.uint8, device=DEV)
    u = torch.rand(k, generator=g, device=DEV)
    return letters[torch.bucketize(u, cdf, out_int32=True, right=True)]


def _starts(lens):
    return torch.cumsum(lens, 0) - lens


def _families(g, n, n_fam, roots_of, alphabet, freqs, subs, indel, indel_mean, with_root=False):
    """n members of n_fam families, family by family: residues (uint8), lengths, family."""
    root_lens = roots_of(g, n_fam)
    roots = _draw(g, alphabet, freqs, int(root_lens.sum()))
    per = torch.full((n_fam,), n // n_fam, dtype=torch.int64, device=DEV)
    per[: n - (n // n_fam) * n_fam] += 1
    fam = torch.repeat_interleave(torch.arange(n_fam, device=DEV), per)
    mlen = root_lens[fam]
    mstart = _starts(mlen)
    total = int(mlen.sum())
    member = torch.repeat_interleave(torch.arange(n, device=DEV), mlen, output_size=total)
    res = roots[(_starts(root_lens)[fam] - mstart)[member] + torch.arange(total, device=DEV)]
    rate = subs[0] + (subs[1] - subs[0]) * torch.rand(n, generator=g, device=DEV)
    ind = torch.full((n,), indel, device=DEV)
    if with_root:  # member 0 of a family is its root
        first = torch.ones(n, dtype=torch.bool, device=DEV)
        first[1:] = fam[1:] != fam[:-1]
        rate[first] = 0.0
        ind[first] = 0.0
    sub = torch.nonzero(torch.rand(total, generator=g, device=DEV) < rate[member]).flatten()
    res[sub] = _draw(g, alphabet, freqs, sub.numel())
    ev = torch.nonzero(torch.rand(total, generator=g, device=DEV) < ind[member]).flatten()
    is_del = torch.rand(ev.numel(), generator=g, device=DEV) < 0.5
    u = torch.rand(ev.numel(), generator=g, device=DEV).clamp_min(1e-7)
    length = 1 + torch.floor(torch.log(u) / math.log(1.0 - 1.0 / indel_mean)).to(torch.int64)
    cover = torch.zeros(total + 1, dtype=torch.int32, device=DEV)
    dels = ev[is_del]
    dend = torch.minimum(dels + length[is_del], (mstart + mlen)[member[dels]])
    one = torch.ones(dels.numel(), dtype=torch.int32, device=DEV)
    cover.index_add_(0, dels, one)
    cover.index_add_(0, dend, -one)
    ins = torch.zeros(total, dtype=torch.int32, device=DEV)
    ins[ev[~is_del]] = length[~is_del].to(torch.int32)
    count = ins + (torch.cumsum(cover[:-1], 0, dtype=torch.int32) == 0)
    lens = torch.zeros(n, dtype=torch.int64, device=DEV)
    lens.index_add_(0, member, count.to(torch.int64))
    out_total = int(lens.sum())
    src = torch.repeat_interleave(torch.arange(total, device=DEV), count, output_size=out_total)
    begin = torch.cumsum(count, 0) - count
    inserted = torch.nonzero(torch.arange(out_total, device=DEV) - begin[src] < ins[src]).flatten()
    out = res[src]
    out[inserted] = _draw(g, alphabet, freqs, inserted.numel())
    return out, lens, fam


def _log_normal(median, lo, hi):
    def roots(g, k):
        z = torch.randn(k, generator=g, device=DEV, dtype=torch.float64)
        return torch.exp(math.log(median) + 0.5 * z).round().clamp(lo, hi).to(torch.int64)
    return roots


def _uniform(g, k, lo, hi):
    return lo + torch.floor(torch.rand(k, generator=g, device=DEV, dtype=torch.float64)
                            * (hi - lo + 1)).to(torch.int64)


def _heavy_tailed(g, k):
    u = torch.rand(k, generator=g, device=DEV)
    out = _log_normal(250, 10, 5_000)(g, k)
    out = torch.where(u >= 0.80, _uniform(g, k, 1_000, 5_000), out)
    return torch.where(u >= 0.99, _uniform(g, k, 5_000, 35_000), out)


def _sequences(g, seqs, n, families):
    """Residues, lengths and family of n sequences in family order."""
    if seqs in ("protein", "protein_close"):
        subs, indel, mean = (((0.05, 0.35), 0.02, 3.0) if seqs == "protein" else
                             ((0.0, 0.04), 0.005, 2.0))
        return _families(g, n, families, _log_normal(300, 50, 1_500), AMINO, AMINO_FREQ, subs,
                         indel, mean)
    if seqs == "mixed":
        return _families(g, n, families, _heavy_tailed, AMINO, AMINO_FREQ, (0.01, 0.50), 0.01,
                         2.0, with_root=True)
    res, lens, fam = _families(g, n, families, lambda g, k: _uniform(g, k, 200, 3_000), NUCLEO,
                               NUCLEO_FREQ, (0.01, 0.10), 0.01, 2.0)
    if seqs == "dna_n":
        res[torch.rand(res.numel(), generator=g, device=DEV) < 0.0005] = ord("N")
    return res, lens, fam


def _pack(res, lens, order):
    """Records in the given order, packed on the device: words, word offsets, lengths."""
    starts, lens = _starts(lens)[order].contiguous(), lens[order]
    words = 1 + 4 * ((lens + 31) // 32)
    offs = _starts(words).contiguous()
    packed = torch.empty(int(words.sum()), dtype=torch.int32, device=DEV)
    lens32 = lens.to(torch.int32).contiguous()
    status = ng.lib().ngia_pack(res.data_ptr(), starts.data_ptr(), lens32.data_ptr(),
                                lens.numel(), offs.data_ptr(), packed.data_ptr(), 0)
    assert status == 0, status
    torch.cuda.synchronize()
    return packed, offs, lens32


def _host(t, dtype, pinned=False):
    if pinned:
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
        h.copy_(t)
        return h.numpy().view(dtype)
    return t.cpu().numpy().view(dtype)


def _database(g, case, seqs, pinned=False):
    """The case's records in index order (length descending) as host arrays."""
    res, lens, fam = _sequences(g, seqs, case["n"], case["families"])
    shuffled = torch.randperm(lens.numel(), generator=g, device=DEV)
    order = shuffled[torch.argsort(-lens[shuffled], stable=True)]
    packed, offs, lens32 = _pack(res, lens, order)
    return (_host(packed, np.uint32, pinned), _host(offs, np.uint64, pinned),
            _host(lens32, np.uint32, pinned))


# ---- the kinds --------------------------------------------------------------------------
EDGES_PER_RECORD = 16  # room in a program's edge buffer (families of ten and chance hits)


def _edge_buffer(n):
    return torch.zeros(n * EDGES_PER_RECORD, 3, dtype=torch.int32, pin_memory=True).numpy()


class _Cluster:
    def __init__(self, g, case):
        self.case = case
        self.edges = _edge_buffer(case["n"])
        self.ctx = ng.Context()
        self.ctx.load(*_database(g, case, case["seqs"]))

    def run(self):
        m, st = self.ctx.group_align(self.case["identity"], self.case["bands"])
        status = ng.lib().ngia_ctx_edges(self.ctx._h, self.edges.ctypes.data, len(self.edges))
        assert status == 0, status
        return self.edges, m, st["candidate_pairs"], st["unique_pairs"]


class _HostLoop:
    def __init__(self, g, case):
        self.case = case
        self.edges = _edge_buffer(case["n"])
        self.db = _database(g, case, case["seqs"], pinned=True)
        self.ctx = ng.Context()

    def run(self):
        m, st = self.ctx.run_host(*self.db, self.case["identity"], self.case["bands"],
                                  self.edges.reshape(-1).view(ng.EDGE_DTYPE))
        return self.edges, m, st["candidate_pairs"], st["unique_pairs"]


class _Fast(_Cluster):
    def run(self):
        self.ctx.sketch_bucket(self.case["bands"])
        return self.ctx.fast_cluster(self.case["identity"], self.case["bands"])


class _Pairs:
    def __init__(self, g, case):
        self.case = case
        m, size = case["pairs"], 5
        a, b = torch.triu_indices(size, size, 1, device=DEV)
        n_fam = max(1, -(-(m // 2) // a.numel()))
        res, lens, fam = _sequences(g, "mixed", n_fam * size, n_fam)
        n = lens.numel()
        order = torch.argsort(-lens, stable=True)
        place = torch.empty_like(order)
        place[order] = torch.arange(n, device=DEV)
        members = place.reshape(n_fam, size)
        related = torch.stack([members[:, a].flatten(), members[:, b].flatten()], 1)[: m // 2]
        i = _uniform(g, m - len(related), 0, n - 1)  # neighbours in length order
        step = _uniform(g, len(i), 1, min(64, n - 1))
        sign = torch.where(torch.rand(len(i), generator=g, device=DEV) < 0.5, -1, 1)
        j = i + sign * step
        j = torch.where((j < 0) | (j >= n), i - sign * step, j)
        j = torch.where((j < 0) | (j >= n), torch.where(i > 0, i - 1, i + 1), j)
        pairs = torch.cat([related, torch.stack([i, j], 1)]).sort(1).values
        pairs = pairs[torch.randperm(m, generator=g, device=DEV)]
        self.pairs = pairs.to(torch.int32).contiguous()
        self.scores = torch.zeros(m, dtype=torch.int32, device=DEV)
        packed, offs, lens32 = _pack(res, lens, order)
        self.ctx = ng.Context()
        self.ctx.load(_host(packed, np.uint32), _host(offs, np.uint64), _host(lens32, np.uint32))

    def run(self):
        self.ctx.align_pairs_device(self.pairs.data_ptr(), len(self.pairs), self.case["identity"],
                                    self.scores.data_ptr())
        return self.scores


class _Raw:
    def __init__(self, g, case):
        self.case = case
        res, lens, fam = _sequences(g, case["seqs"], case["n"], case["families"])
        shuffled = torch.randperm(lens.numel(), generator=g, device=DEV)
        order = shuffled[torch.argsort(-lens[shuffled], stable=True)]
        self.packed, self.offs, self.lens = _pack(res, lens, order)
        n = self.n = case["n"]
        self.sigs = torch.zeros(ng.BANDS, n, dtype=torch.int32, device=DEV)
        self.rep = torch.zeros(ng.BANDS, n, dtype=torch.int32, device=DEV)
        self._sketch_bucket()
        torch.cuda.synchronize()
        rep = self.rep[: case["job_bands"]]  # the jobs of these bands, in the reference's order
        own = torch.arange(n, dtype=torch.int32, device=DEV).expand_as(rep)
        job = rep != own
        self.n_jobs = int(job.sum())
        self.jobs = torch.zeros(rep.numel(), 3, dtype=torch.int32, device=DEV)
        self.jobs[: self.n_jobs, 0] = rep[job]
        self.jobs[: self.n_jobs, 1] = own[job]
        self.edges = torch.zeros_like(self.jobs)
        self.count = torch.zeros(1, dtype=torch.int32, device=DEV)
        torch.cuda.synchronize()

    def _sketch_bucket(self):
        stream = torch.cuda.current_stream().cuda_stream
        ng.sketch(self.packed.data_ptr(), self.offs.data_ptr(), self.n, self.sigs.data_ptr(),
                  stream)
        ng.bucket(self.sigs.data_ptr(), self.n, ng.BANDS, self.rep.data_ptr(), stream)
        return stream

    def run(self):
        stream = self._sketch_bucket()
        ng.align_pairs(self.packed.data_ptr(), self.offs.data_ptr(), self.jobs.data_ptr(),
                       self.n_jobs, self.case["identity"], stream)
        ng.emit_edges(self.jobs.data_ptr(), self.n_jobs, self.edges.data_ptr(),
                      self.count.data_ptr(), stream)
        return self.sigs, self.rep, self.jobs, self.edges, self.count


def _request_sizes(case):
    """Log-uniform sizes, at the middles of equal shares of the distribution."""
    least, ratio, k = case["least"], case["most"] / case["least"], case["requests"]
    return [int(round(least * ratio ** ((i + 0.5) / k))) for i in range(k)]


class _Serve:
    def __init__(self, g, case):
        n = case["n"]
        sizes = _request_sizes(case)
        sizes = [sizes[k] for k in torch.randperm(len(sizes), generator=g, device=DEV).tolist()]
        known = n + sum(s - s // 10 for s in sizes)  # a tenth of the queries are unrelated
        res, lens, fam = _sequences(g, case["seqs"], known, case["families"])
        novel = sum(sizes) - (known - n)
        if novel:
            more, more_lens, _ = _sequences(g, "protein", novel, novel)
            res, lens = torch.cat([res, more]), torch.cat([lens, more_lens])
        perm = torch.randperm(known, generator=g, device=DEV)
        db = perm[:n][torch.argsort(-lens[perm[:n]], stable=True)]
        queries = torch.cat([perm[n:], torch.arange(known, known + novel, device=DEV)])
        queries = queries[torch.randperm(len(queries), generator=g, device=DEV)]
        ctx = ng.Context()
        packed, offs, lens32 = _pack(res, lens, db)
        ctx.load(_host(packed, np.uint32), _host(offs, np.uint64), _host(lens32, np.uint32))
        self.requests, at = [], 0
        for s in sizes:
            packed, offs, lens32 = _pack(res, lens, queries[at:at + s])
            self.requests.append((_host(packed, np.uint32), _host(offs, np.uint64),
                                  _host(lens32, np.uint32)))
            at += s
        self.server = ng.Server(ctx, fam[db].to(torch.int32).cpu().numpy().view(np.uint32),
                                identity=case["identity"], slots=4, max_queries=max(sizes),
                                max_words=max(len(r[0]) for r in self.requests),
                                hbm_budget=8 << 30)
        ctx.close()

    def run(self):
        tickets = [self.server.submit(*r) for r in self.requests]
        return np.concatenate([self.server.wait(t, len(r[2]))[0]
                               for t, r in zip(tickets, self.requests)])


class _Stream:
    def __init__(self, g, case):
        self.case = case
        self.edges = _edge_buffer(case["n"])
        self.db = _database(g, case, case["seqs"], pinned=True)

    def run(self):
        packed, offs, lens = self.db
        m, st = ctypes.c_uint64(), ng.StreamStats()
        status = ng.lib().ngia_stream_graph(
            packed.ctypes.data, packed.size, offs.ctypes.data, lens.ctypes.data, lens.size,
            self.case["identity"], self.case["bands"], self.case["chunk_mib"] << 20,
            self.edges.ctypes.data, len(self.edges), ctypes.byref(m), ctypes.byref(st))
        assert status == 0, status
        return self.edges, m.value, st.candidate_pairs, st.unique_pairs


KINDS = {"cluster": _Cluster, "host": _HostLoop, "fast": _Fast, "pairs": _Pairs, "raw": _Raw,
         "serve": _Serve, "stream": _Stream}


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return KINDS[case["kind"]](g, case)


def run(state):
    return state.run()


def exact(case, seed):
    return None  # whole numbers throughout


def work(case):
    """Bytes of one pass: packed records in (half a byte a residue and the
    offset and length of each), results out.  The arithmetic is 32-bit integer
    and how much of it a pair needs depends on the pair, so no operations are
    counted."""
    kind = case["kind"]
    if kind == "pairs":
        n = case["pairs"] // 2
        return {"bytes": n / 2 * (MEAN_LEN["mixed"] / 2 + 12) + 12 * case["pairs"], "flops": 0}
    if kind == "serve":
        return {"bytes": sum(_request_sizes(case)) * (MEAN_LEN["protein"] / 2 + 12 + 4), "flops": 0}
    n, record = case["n"], MEAN_LEN[case["seqs"]] / 2 + 12
    out = {"cluster": 12, "host": 12, "fast": 4, "stream": 12}.get(kind)
    if kind == "raw":  # signatures, rep rows, jobs and edges
        out = ng.BANDS * 8 + case["job_bands"] * 12
    return {"bytes": n * (record + out), "flops": 0}
