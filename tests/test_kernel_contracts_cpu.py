"""What kernels that begin beside the end of the one before them (csrc/cuda/launch.cuh) have to keep to, checked in the
sources: the faults it prevents come from rare timing, which no run on a GPU shows."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parent.parent / "rannc_b200" / "csrc" / "cuda"


def _source(name):
    """The file without comments."""
    text = re.sub(r"/\*.*?\*/", " ", (CUDA / name).read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _closing(text, start, pair="{}"):
    """Position behind the bracket that closes the one at `start`."""
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def _kernels(name):
    """{kernel: (parameters, body)} of one file."""
    text, out = _source(name), {}
    for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\)\s*)?(\w+)\(", text):
        end = _closing(text, m.end() - 1, "()")
        body = text.index("{", end)
        out[m.group(1)] = (text[m.end():end - 1], text[body:_closing(text, body)])
    return out


# kernels that are launched with launch_after
EARLY = [(f.name, k) for f in sorted(CUDA.glob("*.cu")) for k, (_, body) in _kernels(f.name).items() if "grid_wait()" in body]


def test_every_kernel_that_begins_early_waits():
    text = "".join(_source(f.name) for f in sorted(CUDA.glob("*.cu")))
    names = {k for _, k in EARLY}
    assert {"gemm_tcgen05_kernel", "attn_fwd_kernel", "attn_fwd_persist_kernel", "attn_bwd_kernel", "ln_fwd_kernel"} <= names
    # a launch names the kernel, or a variable that was set to it
    for m in re.finditer(r"launch_after\w*\(\s*(\w+)", text):
        arg = m.group(1)
        sets = set(re.findall(rf"auto {arg}\s*=\s*([^;]+);", text)) or {arg}
        assert all(set(re.findall(r"\w+_kernel", s)) <= names for s in sets), arg


@pytest.mark.parametrize("file,kernel", EARLY)
def test_what_a_kernel_that_begins_early_reads(file, kernel):
    params, body = _kernels(file)[kernel]
    assert not re.search(r"const\s+[\w:]+\s*\*\s*(?:const\s*)?__restrict__", params)
    for text in (body, _source(file), *(_source(h.name) for h in CUDA.glob("*.cuh"))):
        assert not re.search(r"ld\.global(\.\w+)*\.nc\b|\b__ldg\b", text)


@pytest.mark.parametrize("file,kernel", [(f, k) for f, k in EARLY if "tmem_alloc" in _kernels(f)[k][1]])
def test_tensor_memory_is_taken_before_the_next_kernel_may_begin(file, kernel):
    body = _kernels(file)[kernel][1]
    taken = max(m.end() for m in re.finditer(r"tmem_alloc\w*\(", body))
    trigger = [m.start() for m in re.finditer(r"grid_trigger\(\)", body)]
    assert len(trigger) == 1 and trigger[0] > taken
    assert "__syncthreads" in body[taken:trigger[0]]


@pytest.mark.parametrize("file,kernel", [(f, k) for f, k in EARLY if "abort_flag" in _kernels(f)[k][1]])
def test_lanes_of_a_warp_agree_about_a_wait(file, kernel):
    """A wait whose limit runs out ends the work of a whole warp: lanes that went different ways would not meet again at
    the next collective instruction.  Only a role that one lane plays by itself waits by itself."""
    body = _kernels(file)[kernel][1]
    alone = [(m.end() - 1, _closing(body, m.end() - 1)) for m in re.finditer(r"if \(lane == 0\) {", body)]
    for m in re.finditer(r"\bmbar_wait\(", body):
        inside = [body[a:b] for a, b in alone if a < m.start() < b]
        assert inside and not re.search(r"__sync|_sync\(|tmem_|bar_sync|mbar_wait_warp", inside[0])
    # nor does one lane leave a loop that its warp goes through together
    for m in re.finditer(r"if \(issuer\) {", body):
        assert "break" not in body[m.start():_closing(body, m.end() - 1)]
    # a barrier of several warps does not hang on what one of them found
    for m in re.finditer(r"bar_sync_named\(|bar\.sync", body):
        enclosing = [c for c in re.finditer(r"if \(([^{};]*)\) {", body[:m.start()])
                     if _closing(body, c.end() - 1) > m.start()]
        assert not any(re.search(r"\bok\b|mbar_wait", c.group(1)) for c in enclosing)



FAKE_RUNTIME = r"""
#pragma once
#include <cstddef>
#define __device__
#define __forceinline__ inline
typedef int cudaError_t;
typedef void* cudaStream_t;
constexpr cudaError_t cudaSuccess = 0;
struct dim3 { unsigned x, y, z; dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {} };
enum { cudaLaunchAttributeProgrammaticStreamSerialization, cudaLaunchAttributeClusterDimension };
struct cudaLaunchAttribute {
    int id;
    struct { int programmaticStreamSerializationAllowed; struct { unsigned x, y, z; } clusterDim; } val;
};
struct cudaLaunchConfig_t {
    dim3 gridDim, blockDim; size_t dynamicSmemBytes; cudaStream_t stream; cudaLaunchAttribute* attrs; unsigned numAttrs;
};
inline cudaError_t last = 0, next = 0;
inline unsigned clusters = 0;
inline cudaError_t cudaGetLastError() { const cudaError_t e = last; last = 0; return e; }
template <typename... P, typename... A>
cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* c, void (*)(P...), A&&...) {
    clusters = 0;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) clusters = c->attrs[i].val.clusterDim.x;
    if (next) last = next;
    return next;
}
"""
LAUNCHES = r"""
#include "launch.cuh"
void kernel(int) {}
int main() {
    next = 9;   // a launch that fails is reported once
    if (rb::launch_after(kernel, 1, 32, 0, nullptr, 1) != 9 || clusters != 0 || last != 0) return 1;
    if (rb::launch_after_clusters(kernel, 2, 2, 32, 0, nullptr, 1) != 9 || clusters != 2 || last != 0) return 2;
    next = 0, last = 7;   // what somebody else left is theirs to find
    if (rb::launch_after(kernel, 1, 32, 0, nullptr, 1) != 0 || last != 7) return 3;
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_a_failed_launch_is_reported_once(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE_RUNTIME)
    (tmp_path / "launches.cpp").write_text(LAUNCHES)
    exe = str(tmp_path / "launches")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(tmp_path), "-I", str(CUDA), str(tmp_path / "launches.cpp"), "-o",
                    exe], check=True)
    assert subprocess.run([exe]).returncode == 0
    # every result is looked at, and launches with these attributes go through these functions
    for f in sorted(CUDA.glob("*.cu")):
        text = _source(f.name)
        assert all(text[:m.start()].rstrip()[-1] not in ";{}" for m in re.finditer(r"\blaunch_after\w*\(", text)), f.name
        assert "cudaLaunchKernelEx" not in text, f.name


# ------------------------------------------------------------------------- barriers of the attention backward
# The roles of one block run at any speed relative to each other.  Their loops over the query blocks are read from the
# source as sequences of barrier operations, products and loads; the table says under which condition block i does one,
# which barrier of an array it means and which phase of it.  A wait looks at a phase's parity alone: it is passed when the
# number of phases that have ended is odd or even as it should be.
STAGES = 3
TOKEN = re.compile(r"mbar_(wait)(?:_warp)?\(&?(\w+)|mbar_(arrive)\(&?(\w+)|umma_(commit)\(&?(\w+)|"
                   r"umma_f16\w*\(tmem \+ (C_)(\w+)|(load_qd|put_stats)\((i)")
_always = lambda i, nq: True                       # noqa: E731
_reload = lambda i, nq: i >= 1 and i + 2 < nq      # noqa: E731
RULES = {   # (role, what, barrier): (condition, index in an array, phase that is waited for)
    ("load", "wait", "qd_full"): (_always, lambda i: i % STAGES, lambda i: i // STAGES),
    ("load", "wait", "s_free"): (lambda i, nq: i > 0, None, lambda i: i - 1),
    ("load", "commit", "s_full"): (_always, None, None),
    ("load", "wait", "p_done"): (_reload, None, lambda i: i - 1),
    ("load", "wait", "qd_free"): (_reload, lambda i: (i + 2) % STAGES, lambda i: (i - 1) // STAGES),
    ("load", "load_qd", "i"): (_reload, None, None),
    ("grad", "wait", "qd_full"): (_always, lambda i: i % STAGES, lambda i: i // STAGES),
    ("grad", "wait", "pds_ready"): (_always, None, lambda i: i),
    ("grad", "wait", "dq_taken"): (lambda i, nq: i > 0, None, lambda i: i - 1),
    ("grad", "commit", "ds_done"): (_always, None, None),
    ("grad", "commit", "qd_free"): (lambda i, nq: i + STAGES < nq, lambda i: i % STAGES, None),
    ("grad", "commit", "p_done"): (_always, None, None),
    ("drain", "wait", "ds_done"): (_always, None, lambda i: i),
    ("drain", "arrive", "dq_taken"): (_always, None, None),
    ("drain", "put_stats", "i"): (lambda i, nq: i + 2 < nq, lambda i: i & 1, None),
    ("drain", "arrive", "dq_free"): (_always, None, None),
    ("drain", "wait", "dq_free"): (_always, None, lambda i: i),
    ("drain", "arrive", "dq_ready"): (_always, None, None),
    ("drain", "wait", "dq_ready"): (_always, None, lambda i: i),
    ("math", "wait", "stats_full"): (_always, lambda i: i & 1, lambda i: i >> 1),
    ("math", "wait", "s_full"): (_always, None, lambda i: i),
    ("math", "arrive", "s_free"): (_always, None, None),
    ("math", "wait", "ds_done"): (lambda i, nq: i > 0, None, lambda i: i - 1),
    ("math", "wait", "p_done"): (lambda i, nq: i > 0, None, lambda i: i - 1),
    ("math", "arrive", "pds_ready"): (_always, None, None),
}


def _bwd_roles():
    """{role: [(what, barrier)]} of the loops over the query blocks."""
    body = _kernels("attn_bwd.cu")["attn_bwd_kernel"][1]
    start = body.index("if (warp == LOAD_WARP) {", body.index("grid_wait()"))
    out = {}
    for role in ("load", "grad", "drain", "math"):
        open_ = body.index("{", start)
        section = body[open_:_closing(body, open_)]
        start = open_ + len(section)
        loops = [m for m in re.finditer(r"for \(int i = 0; i < nq[^)]*\)\s*{", section)]
        assert len(loops) == 1, role
        loop = section[loops[0].start():_closing(section, loops[0].end() - 1)]
        out[role] = [tuple(x for x in m.groups() if x) for m in TOKEN.finditer(loop)]
    return out


def _programs(nq):
    """{actor: [step]}; products and the commits behind them are steps of a queue that the tensor core works off."""
    progs = {a: [] for a in ("load", "grad", "drain", "math", "load queue", "grad queue")}
    progs["load"] += [("put", i % STAGES, i) for i in range(min(STAGES, nq))]
    progs["drain"] += [("arrive", ("stats_full", i & 1)) for i in range(min(2, nq))]
    for role, tokens in _bwd_roles().items():
        for i in range(nq):
            for what, name in tokens:
                if what == "C_":
                    progs[role + " queue"].append(("read", None if name == "DQ" else (i % STAGES, i), len(progs[role])))
                    continue
                when, index, phase = RULES[role, what, name]
                if not when(i, nq):
                    continue
                bar = (name, index(i) if index else 0)
                if what == "wait":
                    progs[role].append(("wait", bar, phase(i)))
                elif what == "commit":
                    progs[role + " queue"].append(("arrive", bar, len(progs[role])))
                elif what == "load_qd":
                    progs[role].append(("put", (i + 2) % STAGES, i + 2))
                else:
                    progs[role].append(("arrive", ("stats_full", i & 1) if what == "put_stats" else bar))
    return progs


@pytest.mark.parametrize("nq", [1, 2, 3, 4, 5, 7])
def test_attention_backward_roles_at_any_speed(nq):
    progs = _programs(nq)
    actors = list(progs)
    # how often each barrier has ended a phase, and what each stage holds, by the position of an actor
    arrived = {a: [{}] for a in actors}
    held = [{}]
    for a in actors:
        for step in progs[a]:
            count = dict(arrived[a][-1])
            if step[0] == "arrive":
                count[step[1]] = count.get(step[1], 0) + 1
            if step[0] == "put":
                held.append({**held[-1], step[1]: step[2]})
                count["qd_full", step[1]] = count.get(("qd_full", step[1]), 0) + 1
            elif a == "load":
                held.append(held[-1])
            arrived[a].append(count)

    def ended(bar, at):
        return sum(arrived[a][pc].get(bar, 0) for a, pc in zip(actors, at))

    seen, todo = set(), [(0,) * len(actors)]
    while todo:
        at = todo.pop()
        if at in seen:
            continue
        seen.add(at)
        moves = 0
        for k, a in enumerate(actors):
            if at[k] == len(progs[a]):
                continue
            step = progs[a][at[k]]
            if step[0] == "wait":
                n = ended(step[1], at)
                if (n - step[2]) % 2 == 0:
                    continue
                assert n == step[2] + 1, f"{a} passes {step} with {n} phases ended"
            elif a.endswith("queue"):
                if at[actors.index(a.split()[0])] < step[2]:
                    continue   # not issued yet
                if step[0] == "read" and step[1]:
                    assert held[at[actors.index("load")]].get(step[1][0]) == step[1][1], f"{step} reads another block"
            moves += 1
            todo.append(at[:k] + (at[k] + 1,) + at[k + 1:])
        assert moves or all(pc == len(progs[a]) for a, pc in zip(actors, at)), \
            "stuck before " + ", ".join(str(progs[a][pc]) for a, pc in zip(actors, at) if pc < len(progs[a]))
    assert len(seen) > nq


# ------------------------------------------------------------------------- what a product is asked for
@pytest.mark.parametrize("deterministic", [False, True])
def test_partitioned_weight_gradient_passes_the_order_on(deterministic, monkeypatch):
    """A tensor-partitioned linear's weight gradient asks for tiles that are summed whole under
    torch.use_deterministic_algorithms, like every other product."""
    import torch

    from rannc_b200.ops import _lib
    from rannc_b200.parallel import distop

    seen = []

    class Fake:
        @staticmethod
        def rb_gemm(args, stream):
            seen.append(args._obj.in_order)
            return 0

    monkeypatch.setattr(_lib, "lib", lambda: Fake)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: None)
    before = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(deterministic)
    try:
        distop._gemm_rs(torch.zeros(16, 8, dtype=torch.bfloat16), torch.zeros(16, 8, dtype=torch.bfloat16), 8, 8, [4096], 8,
                        1.0)
    finally:
        torch.use_deterministic_algorithms(before)
    assert seen == [int(deterministic)]


# tiles of 256 x 256 on 74 pairs of SMs
@pytest.mark.parametrize("m,n,K,how", [
    (8, 9, 8192, 0), (2, 37, 8192, 0),                                         # no last wave
    (8, 11, 448, 0), (8, 11, 512, 2), (8, 11, 1024, 4), (8, 11, 4096, 5),      # 1 + 14
    (2, 49, 1024, 3), (11, 9, 1024, 0), (11, 9, 1536, 2),                      # 1 + 24, 1 + 25
    (10, 11, 1024, 0), (10, 11, 1536, 2), (3, 37, 1536, 2),                    # 1 + 36, 1 + 37
    (16, 16, 1024, 0), (16, 16, 1536, 2), (120, 4, 512, 0), (120, 4, 1024, 0), (120, 4, 2048, 2),   # 3 + 34, 6 + 36
    (7, 16, 1024, 0), (7, 16, 1536, 1), (8, 17, 4096, 1), (8, 17, 2048, 0),    # 1 + 38, 1 + 62
    (6, 23, 16384, 0), (12, 18, 16384, 0), (12, 12, 16384, 0), (3, 49, 16384, 0)])   # 1 + 64, 2 + 68, 1 + 70, 1 + 73
def test_which_last_waves_are_shared_out(m, n, K, how):
    from rannc_b200.ops.gemm import last_wave

    assert last_wave(256 * m, 256 * n - 100, K) == how
    assert last_wave(256 * m, 256 * n - 100, K, in_order=True) == 0
