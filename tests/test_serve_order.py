"""The serving loop hands list nodes from lane to lane: a block's link and value
are written by the lane that allocated it and read by the lane that owns the
job.  Votes and shuffles order no memory, so on every way from the writes to
the walk there has to be a barrier of the warp: one at the step's own level,
in no loop or branch.  Checked on the source, since a missing barrier shows
on the GPU only by chance."""
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SERVE = os.path.join(ROOT, "halloc_b200", "csrc", "ha_serve.cu")


def _statements(text):
    """(statement, brace depth) of the kernel's source without its comments."""
    out, depth = [], 0
    for line in text.split("\n"):
        line = line.split("//")[0]
        for part in line.replace("{", "\n{\n").replace("}", "\n}\n").split("\n"):
            part = part.strip()
            if part == "{":
                depth += 1
            elif part == "}":
                depth -= 1
            elif part:
                out.append((part, depth))
    return out


def test_a_barrier_lies_between_the_writes_and_the_walk():
    with open(SERVE) as f:
        text = f.read()
    st = _statements(text[text.index("ha_serve_k(ServeParams P)"):])
    first = next(i for i, (s, _) in enumerate(st) if s.startswith("for (;;)"))
    level = next(d for s, d in st[first + 1:])  # the depth of the step's own statements
    written = max(i for i, (s, _) in enumerate(st) if "reinterpret_cast<uint32_t *>(p)[2] =" in s)
    walked = min(i for i, (s, _) in enumerate(st) if "reinterpret_cast<const uint32_t *>(head)[2]" in s)
    assert first < written < walked
    between = [s for s, d in st[written:walked] if d == level]
    assert "__syncwarp();" in between
