"""Rules that the kernels' source has to keep and that no run on a GPU would show broken."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "csrc" / "kernels"
SOURCES = sorted(p for p in KERNELS.iterdir() if p.suffix in (".cu", ".cuh"))
WAIT = re.compile(r"\b(?:mbar_wait|mbar_wait_abortable|PS_WAIT|PR_WAIT|WALK_WAIT)\(")


def _code(path):
    """The source without comments, directives and macro bodies, its lines kept."""
    text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m[0].count("\n"), path.read_text(), flags=re.S)
    lines, macro = [], False
    for line in (re.sub(r"//.*", "", line) for line in text.split("\n")):
        skip = macro or line.lstrip().startswith("#")
        macro = skip and line.rstrip().endswith("\\")
        lines.append("" if skip else line)
    return "\n".join(lines)


def _statements(code):
    """(line, text, headers of the blocks around it) of every statement."""
    blocks, start, depth = [], 0, 0
    for i, ch in enumerate(code):
        if ch in "()":
            depth += 1 if ch == "(" else -1
        elif ch == "{" and (depth == 0 or code[:i].rstrip().endswith(")")):
            blocks.append((code[start:i].strip(), depth))
            start, depth = i + 1, 0
        elif ch == "}" and depth == 0:
            if blocks:
                depth = blocks.pop()[1]
            start = i + 1
        elif ch == ";" and depth == 0:
            text = code[start:i]
            lead = len(text) - len(text.lstrip())
            yield code.count("\n", 0, start + lead) + 1, text.strip(), [b for b, _ in blocks]
            start = i + 1


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_warps_agree_on_waits_that_may_give_up(path):
    """A bounded wait is answered lane by lane.  Where a warp goes on as a whole (it meets at a
    __syncwarp, votes, or signals for all its lanes), lanes that gave up and lanes that did not must
    not part: the answers are voted on, in the statement of the wait or in the next one."""
    one = re.compile(r"lane == 0|threadIdx\.x == 0|tid == 0|\bt == 0|leader")
    code, wrong = _code(path), []
    statements = list(_statements(code))
    for n, (line, text, blocks) in enumerate(statements):
        if not WAIT.search(text) or "inline__" in text:
            continue
        if any(one.search(b) for b in blocks) or one.search(text.split("wait")[0]):
            continue
        follows = statements[n + 1][1] if n + 1 < len(statements) else ""
        # the drain at a role's end asks for no answer
        answered = re.search(r"=|return|if", WAIT.split(text)[0].rsplit(")", 1)[-1])
        if answered and "_all_sync(" not in text + follows and "warp_all(" not in text + follows:
            wrong.append(f"{path.name}:{line}: {' '.join(text.split())[:90]}")
    assert not wrong, "\n".join(wrong)


@pytest.mark.parametrize("name", ["gemm_walk.cu", "gemv.cu"])
def test_rings_that_bulk_copies_refill_are_handed_back_behind_their_reads(name):
    """A warp that reads a slab into registers gives it back through hand_back, whose arrival
    depends on what was read."""
    code = _code(KERNELS / name)
    assert re.search(r"hand_back\(&(c_)?empty\[", code)
    assert not re.search(r"mbar_arrive\(&(c_)?empty\[", code)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_copies_in_flight_are_waited_for_on_barriers_of_their_own(path):
    """Before a copying warp leaves, it waits for what it has in flight, without a look at the abort
    word: on barriers with one arrival, its own, so that the bytes alone complete them."""
    code = _code(path)
    for kernel in re.split(r"__global__", code)[1:]:
        counts = dict(re.findall(r"mbar_init\(&?(\w+)(?:\[\w+\])?, (.+?)\);", kernel))
        names = re.findall(
            r"(?:for \([^;]*;[^;]*;[^;{]*\)|if \(.*\))\s+mbar_wait\(&(\w+)\[", kernel)
        for name in names:
            alias = re.search(r"uint64_t\* " + name + r" = (.+?);", kernel)
            owners = [name] if name in counts else re.findall(r"\w+", alias[1])
            for count in (counts[o] for o in owners if o in counts):
                assert count == "1" or re.fullmatch(r"FMT == 0 \? 1 : .+", count), (name, count)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_whole_warps_arrive_at_cluster_barriers(path):
    """The cluster barrier is of the aligned form, which every lane of a warp executes together: no
    branch that lanes may take apart lies between it and the barrier or __syncwarp before it."""
    for part in _code(path).split("cluster_sync_all();")[:-1]:
        code = re.split(r"__sync(?:threads|warp)\(\);", part)[-1]
        assert code != part, path.name
        whole = re.compile(r"warp == \d|SPLIT")
        apart = [c for c in re.findall(r"\bif \((.*?)\)", code) if not whole.fullmatch(c)]
        assert not apart and not re.search(r"\b(for|while)\b", code), (path.name, code[-300:])


def _closing(code, at):
    """Index behind the bracket that closes the one at `at`."""
    pairs, depth = {"(": 1, ")": -1, "{": 1, "}": -1}, 0
    for i in range(at, len(code)):
        depth += pairs.get(code[i], 0)
        if depth == 0:
            return i + 1
    raise ValueError(code[at:at + 80])


def _functions(code):
    """(kind, name, parameters, body) of every function of the source."""
    for word in ("__launch_bounds__", "__cluster_dims__"):
        while word + "(" in code:
            at = code.index(word + "(")
            code = code[:at] + code[_closing(code, at + len(word)):]
    for m in re.finditer(r"__(global|device)__\s[^;({=]*?(\w+)\(", code):
        end = _closing(code, m.end() - 1)
        tail = re.match(r"\s*(const\s*)?\{", code[end:])
        if tail:                                                   # not a declaration
            body = end + tail.end() - 1
            yield m[1], m[2], code[m.end():end - 1], code[body:_closing(code, body)]


def test_kernels_that_start_early_load_through_the_coherent_path():
    """A kernel that is resident while the ones in front of it still write must not read what they
    write through the read-only path, nor let the compiler move a load ahead of its grid_wait: no
    __ldg, and no __restrict__ on what it reads.  The decode tables are constant from start-up on."""
    both = {"resid", "state", "hist", "partial", "tickets", "ws"}   # read and written
    plainly = {"gdn_chunk_kernel"}                                  # waits, but is not launched early
    early, wrong = 0, []
    for path in SOURCES:
        functions = list(_functions(_code(path)))
        waits = lambda body: "grid_wait()" in body or "early.load(" in body
        if path.suffix == ".cuh" or not any(waits(body) for *_, body in functions):
            continue
        for kind, name, parameters, body in functions:
            if name in plainly or kind == "global" and not waits(body):
                continue
            early += kind == "global"
            for p in re.split(r",\s*", parameters):
                read = re.search(r"const (\w+)(?:<\w+>)?\* __restrict__", p)
                if (read and not read[1].startswith("E8p")) or (
                        "__restrict__" in p and p.split()[-1] in both):
                    wrong.append(f"{path.name}: {name}: {' '.join(p.split())}")
            if "__ldg(" in body:
                wrong.append(f"{path.name}: {name}: __ldg")
    assert early > 25
    assert not wrong, "\n".join(wrong)
