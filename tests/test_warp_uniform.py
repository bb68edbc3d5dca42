"""A warp of the solver may only branch as a whole on what other warps change meanwhile.

Between a branch and a collective of all 32 lanes (a shuffle, a vote, a reduction) every lane has to take the same way.
A value that each lane reads for itself with vload may differ from lane to lane while another warp writes it, so a
decision about it is made in one lane and handed out (vload_warp, a vote), or nothing after it is a collective.  This
reads fdgpu_kernels.cu: in every function that contains a collective, directly or through a call, no condition on a
vload, or on a variable set from one, may lead to a return, break, continue, goto or collective, except in code that single
lanes run."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtomoc_gb300", "csrc", "fdgpu_kernels.cu")
OWN_READ = r"\bvload\("
LANES = re.compile(r"\b(lane|tid)\s*(==|<)|threadIdx\.x & 31\)\s*==")
JUMP = re.compile(r"\b(return|break|continue|goto)\b")


def matching(s, i):
    """index after the bracket that closes the one at s[i]"""
    pair = {"(": ")", "{": "}"}[s[i]]
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == s[i]) - (s[k] == pair)
        if depth == 0:
            return k + 1
    raise ValueError(s[i:i + 60])


def statement(s, i):
    """end of the statement that starts at s[i]"""
    while s[i].isspace():
        i += 1
    if s[i] == "{":
        return matching(s, i)
    m = re.match(r"(if|for|while)\s*\(", s[i:])
    if m:
        end = statement(s, matching(s, i + m.end() - 1))
        e = re.match(r"\s*else\b", s[end:])
        return statement(s, end + e.end()) if m.group(1) == "if" and e else end
    while s[i] != ";":
        i = matching(s, i) if s[i] in "({" else i + 1
    return i + 1


def functions(text):
    for m in re.finditer(r"^[\w:&*<> ,]*?\b(\w+)\([^;{}]*?\)\n\{", text, re.M):
        yield m.group(1), text[m.end() - 1:matching(text, m.end() - 1)]


def is_collective(names):
    calls = "|".join(sorted(names)) or "(?!)"
    return re.compile(r"_sync\(0xffffffffu|\b(" + calls + r")\(")


def violations(text):
    text = re.sub(r"/\*.*?\*/|//[^\n]*", " ", text, flags=re.S)
    text = re.sub(r"^#.*$", "", text, flags=re.M)
    body = dict(functions(text))
    wide = set()
    while True:
        more = {n for n, b in body.items() if is_collective(wide).search(b)} - {"vload_warp"}
        if more == wide:
            break
        wide = more
    coll = is_collective(wide | {"vload_warp"})
    found = []

    def walk(name, s, own):
        i = 0
        while i < len(s):
            m = re.compile(r"\b(if|while|for)\s*\(|\b(\w+) = ([^;]*);").search(s, i)
            if not m:
                return
            if m.group(2):
                if re.search(OWN_READ, m.group(3)) and "_sync(" not in m.group(3):
                    own.add(m.group(2))
                i = m.start() + len(m.group(2))
                continue
            end = matching(s, m.end() - 1)
            cond, stop = s[m.end() - 1:end], statement(s, end)
            controlled = s[end:stop]
            reads = re.search(OWN_READ, re.sub(r"_(any|all|ballot)_sync\(.*", "", cond)) or any(re.search(r"\b%s\b" % v, cond) for v in own)
            if not LANES.search(cond):
                # a collective later in the condition itself is reached by some lanes only, too
                if reads and (JUMP.search(controlled) or coll.search(controlled) or coll.search(re.sub(r".*?vload\(", "", cond, count=1))):
                    found.append((name, cond))
                walk(name, controlled, own)
            i = stop

    for name in wide:
        if name in body:
            walk(name, body[name][1:], set())
    return wide, found


def test_finds_what_it_is_for():
    bad = "__device__ bool f(int a)\n{\n    if (vload(x) > a) return true;\n    return __any_sync(0xffffffffu, a);\n}\n"
    good = bad.replace("vload(x)", "vload_warp(x)")
    by_name = bad.replace("if (vload(x) > a)", "const int v = vload(x);\n    if (v > a)")
    one_lane = bad.replace("if (vload(x) > a) return true;", "if (lane == 0 && vload(x) > a) y = 1;")
    assert violations(bad)[1] and violations(by_name)[1]
    assert not violations(good)[1] and not violations(one_lane)[1]


def test_warps_branch_as_a_whole():
    wide, found = violations(open(SRC).read())
    assert {"warp_chunk", "graph_release", "scan_open", "keys_above", "exit_floor", "resume_graph", "resume_waiter", "run_walk"} <= wide
    assert not found, found
