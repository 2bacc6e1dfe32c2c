"""What the kernels' sources have to say so that programmatic dependent launch is sound, read on the CPU.

A kernel that waits for the kernel before it (`grid_dependency_wait`) reads that kernel's results behind the wait.  A pointer
declared `__restrict__` lets the compiler move a load through it in front of the wait, so only two kinds of parameters
may be declared so: `const` ones that no kernel of a step writes, and ones that the kernel only stores through."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libllm_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))

# weights, biases and tables, by the name of the parameter ("kernel.name" where the name means something else elsewhere)
FIXED = set("""table pos_table weight bias conv conv_w w2 w0 a_bias norm_w q_norm k_norm null_scores temp col_scale col_bias a2 g2 dt_bias
a_log w_uk w_uv q_weight kv_weight W up down mu skip w_dt bias_i bias_f mix outw inw bonus_pack_kernel.u""".split())
STEP = {"moe_rows_kernel.weight", "moe_identity_kernel.weight", "moe_grouped_kernel.weight", "moe_gather_kernel.weight", "moe_tc_kernel.weight"}
# results of a kernel that it does not read
STORED = set("""out dst q_out kcache vcache prep gate cq_out cache c_out kr_out xs mid C rec scal vals den resid_out
attention_decode_kernel.ws_o attention_decode_kernel.ws_ml latent_decode_kernel.ws_o latent_decode_kernel.ws_ml""".split())
READ_TOO = {"sample_kernel.out"}


def closing(text, at, pair):
    depth = 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[at], 0)
        at += 1
    return at


def split(params):
    out, depth, cur = [], 0, ""
    for c in params:
        depth += (c in "<([") - (c in ">)]")
        if c == "," and depth == 0:
            out.append(cur.strip())
            cur = ""
        else:
            cur += c
    return out + [cur.strip()] if cur.strip() else out


def functions(path):
    """(name, parameters, body, is a kernel) of every kernel and device function of a source file."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__global__|__device__", text):
        at = m.end()
        while True:
            call = re.compile(r"([A-Za-z_]\w*)\s*\(|[;{=]").search(text, at)
            if call is None or call.group(1) is None:          # a variable
                break
            end = closing(text, call.end(), "()")
            if call.group(1).startswith("__"):                  # __launch_bounds__(..)
                at = end
                continue
            rest = text[end:].lstrip()
            if rest.startswith("{"):
                start = text.index("{", end)
                yield call.group(1), split(text[call.end():end - 1]), text[start:closing(text, start + 1, "{}")], m.group(0) == "__global__"
            break


KERNELS = [(os.path.basename(f), *k) for f in FILES for k in functions(f)]


def test_the_sources_are_read():
    waiting = [k for k in KERNELS if k[4] and "grid_dependency_wait" in k[3]]
    assert len(waiting) >= 80 and len([k for k in KERNELS if not k[4]]) >= 60


@pytest.mark.parametrize("file", sorted({k[0] for k in KERNELS}))
def test_no_load_may_leave_the_wait_behind(file):
    wrong = []
    for _, name, params, body, kernel in (k for k in KERNELS if k[0] == file):
        if kernel and "grid_dependency_wait" not in body:
            continue                                            # launched behind its predecessor's end
        for p in params:
            if "__restrict__" not in p:
                continue
            arg = re.sub(r".*[*\s]", "", p)
            full = f"{name}.{arg}"
            if p.startswith("const"):
                ok = (arg in FIXED or full in FIXED) and full not in STEP or not kernel and arg == "w"
            else:
                ok = (arg in STORED or full in STORED) and full not in READ_TOO or not kernel and arg == "o"
            if not ok:
                wrong.append(f"{full}: {p}")
        if kernel and re.search(r"__ldg\s*\(", body):
            wrong.append(f"{name}: __ldg")
    assert not wrong, "\n".join(wrong)


def test_loads_from_tensor_memory_are_waited_for_where_they_are_issued():
    """What `tcgen05.ld` writes is undefined until the wait: between the two a register may not even be copied, which a compiler does where
    the load's block ends (a loop's back edge, an if).  So the wait follows in the same block, and a load with its wait is one statement."""
    text = open(os.path.join(CSRC, "tc_common.cuh")).read()
    one = text[text.index("void tc_ld16(unsigned"):]
    assert re.search(r"asm volatile\([^;]*tcgen05\.ld[^)]*?tcgen05\.wait::ld", one[:one.index("\n}\n")], re.S)
    loads = 0
    for file, name, _, body, _ in KERNELS:
        for m in re.finditer(r"tc_ld16_issue\(", body):
            if name == "tc_ld16_issue":
                continue
            loads += 1
            line = body[body.rfind("\n", 0, m.start()) + 1:m.start()]
            assert not re.search(r"\bif\b", line), f"{file}: {name}: a load that is issued or not"
            at, depth = m.end(), 0
            while not body.startswith("tc_ld_wait()", at):
                depth += {"{": 1, "}": -1}.get(body[at], 0)
                assert depth >= 0, f"{file}: {name}: the block ends before the wait"
                at += 1
    assert loads >= 10


def calls(body, names):
    """Where a body first calls one of these functions."""
    return min((m.start() for m in re.finditer(r"\b(\w+)\s*(?:<[^;()]*>)?\(", body) if m.group(1) in names), default=None)


def test_no_shared_memory_of_another_cta_is_touched_before_the_cluster_is_known_to_run():
    """A CTA of a cluster may touch another one's shared memory only behind a cluster barrier that both have come to: until then that CTA need not be there."""
    remote = {name for _, name, _, body, kernel in KERNELS if not kernel and "mapa" in body}
    barrier = {name for _, name, _, body, kernel in KERNELS if not kernel and "barrier.cluster.wait" in body}
    for _ in range(2):                                          # and what is made of them
        barrier |= {name for _, name, _, body, kernel in KERNELS if not kernel and calls(body, barrier) is not None}
        remote |= {name for _, name, _, body, kernel in KERNELS if not kernel and calls(body, remote) is not None}
    seen, wrong = 0, []
    for file, name, _, body, kernel in KERNELS:
        first = calls(body, remote) if kernel else None
        if first is not None:
            seen += 1
            known = calls(body, barrier)
            if known is None or known > first:
                wrong.append(f"{file}: {name}")
    assert seen >= 3 and not wrong, (seen, wrong)
