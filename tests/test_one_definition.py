"""Names with external linkage are defined in one translation unit: two files that define the
same class or function of namespace vlt break the one-definition rule as soon as one body is
not inlined, and the linker then keeps either."""
import collections
import glob
import os
import re

from violet_gb300 import build


def definitions(path):
    """(name, signature) of the classes and functions that a source defines in named
    namespaces without `static`."""
    text = open(path).read()
    text = re.sub(r"//[^\n]*|/\*.*?\*/", " ", text, flags=re.S)
    text = re.sub(r'"(?:\\.|[^"\\\n])*"', '""', text)
    text = re.sub(r"^[ \t]*#(?:[^\n]*\\\n)*[^\n]*", "", text, flags=re.M)
    out, stack, start = [], [], 0
    for m in re.finditer(r"[{};]", text):
        head = " ".join(text[start:m.start()].split())
        start = m.end()
        if m.group() == "}":
            stack.pop()
        elif m.group() == "{":
            ns = re.search(r'(?:^|\s)namespace\s*([\w:]*)$', head)
            if ns or head == 'extern ""':
                stack.append("anonymous" if ns and not ns.group(1) else "named")
                continue
            if all(s == "named" for s in stack) and not re.search(r"\bstatic\b", head):
                kind = re.search(r"\b(?:struct|class|union|enum)\s+(\w+)\s*(<[^:]*>)?\s*(?::[^:].*)?$", head)
                fn = re.search(r"(\w+)\s*(\(.*\))\s*(?:const)?$", head)
                if kind and "(" not in head:
                    out.append((kind.group(1), kind.group(2) or ""))
                elif fn:
                    out.append((fn.group(1), fn.group(2)))
            stack.append("other")
    assert not stack, path
    return out


def test_one_definition():
    where = collections.defaultdict(set)
    sources = sorted(glob.glob(os.path.join(build.CSRC, "*.cu")))
    assert len(sources) == len(build.SOURCES)
    for path in sources:
        found = definitions(path)
        assert found, path
        for d in found:
            where[d].add(os.path.basename(path))
    assert any(n == "launch_hg_select" for n, _ in where) and any(n == "DnTemporalF" for n, _ in where)
    assert not {d: f for d, f in where.items() if len(f) > 1}
