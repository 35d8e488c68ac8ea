"""Ordering rules of kernels that run beside others, checked on their source: what a
race does on a GPU cannot be made to happen at will, so the rules are checked where they are written."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pbpic_b200", "csrc")


def source(name):
    """A source file without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def functions(text):
    """Bodies of the functions defined in a source, by name (overloads joined)."""
    out = {}
    for m in re.finditer(r"\b(\w+)\s*\([^;{}()]*(?:\([^;{}()]*\)[^;{}()]*)*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        if m.group(1) not in ("if", "for", "while", "switch"):
            out[m.group(1)] = out.get(m.group(1), "") + text[m.end():i]
    return out


def clearing_steps():
    """k_fused_tables' accesses to the chunks' totals in program order: S a block leaves its total, F
    a fence, A it counts itself, C the last one counted clears the words."""
    body = functions(source("kernels_sort.cuh"))["k_fused_tables"]
    ops = {"S": r"totals\[chunk\]\s*=", "F": r"__threadfence\(\)", "A": r"atomicAdd\(&words\[0\]", "C": r"words\[k\]\s*=\s*0"}
    return [op for _, op in sorted((m.start(), op) for op, rx in ops.items() for m in re.finditer(rx, body))]


def left_over(steps, blocks=2):
    """Whether some order of `blocks` running `steps` ends with a word that is not zero. A store (S, C) lands at any time
    after it is issued, at the latest at its block's next fence or at the end."""
    seen = set()

    def run(pc, pending, words, count, last):
        state = (pc, pending, words, count, last)
        if state in seen:
            return False
        seen.add(state)
        if not pending and all(p == len(steps) for p in pc):
            return any(words)
        for k, (_, word, value) in enumerate(pending):  # a store in flight lands
            w = words[:word] + (value,) + words[word + 1:]
            if run(pc, pending[:k] + pending[k + 1:], w, count, last):
                return True
        for b in range(blocks):
            if pc[b] == len(steps):
                continue
            op, nxt = steps[pc[b]], pc[:b] + (pc[b] + 1,) + pc[b + 1:]
            if op == "F" and any(p[0] == b for p in pending):
                continue  # the fence waits for the block's stores
            if op == "S":
                args = pending + ((b, b, 1),), words, count, last
            elif op == "A":
                args = pending, words, count + 1, b if count == blocks - 1 else last
            elif op == "C" and last == b:
                args = pending + tuple((b, k, 0) for k in range(blocks)), words, count, last
            else:
                args = pending, words, count, last
            if run(nxt, *args):
                return True
        return False

    return run((0,) * blocks, (), (0,) * blocks, 0, None)


def test_chunk_totals_are_clear_after_every_launch():
    """A total that lands after its word was cleared would be taken for one of the next launch."""
    assert left_over(["S", "A", "C"])  # (the model finds it)
    steps = clearing_steps()
    assert [s for s in steps if s != "F"] == ["S", "A", "C"]
    assert not left_over(steps)
    at = steps.index("A")  # the fence after the count: nothing of the clearing is issued ahead of it
    assert steps[at - 1] == "F" and steps[at + 1] == "F"


def test_early_launches_load_coherently():
    """A kernel that starts under the one before it (launch_early) must not read through the
    non-coherent path, which is for memory that nothing writes while the kernel lives."""
    api = source("pbpic_api.cu")
    early = set(re.findall(r"launch_early\((k_\w+)", api))
    assert early == {"k_fused_tables", "k_fused_perm"}
    bodies = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cuh"):
            for k, body in functions(source(name)).items():
                bodies[k] = bodies.get(k, "") + body
    reached, todo = set(), list(early)
    while todo:  # the kernels and every device function they call
        k = todo.pop()
        if k not in reached:
            reached.add(k)
            todo += [c for c in re.findall(r"\b(\w+)\s*(?:<[^;<>()]*>)?\(", bodies[k]) if c in bodies]
    assert {"chunk_counts", "chunk_tables", "fused_count", "fused_slots", "perm_tile"} <= reached
    for k in reached:
        assert "cudaGridDependencySynchronize" in bodies[k] or k not in early, k
        assert not re.search(r"__ldg\(|\bldg_part\(|\.nc\b", bodies[k]), k
