"""Models of kernel handshakes whose failure would be a hang: every interleaving of the warps is explored on the CPU."""

import itertools
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "cosmos_predict25_b200" / "ops" / "csrc"


def explore(start, successors):
    """All reachable states, and those from which nothing can happen."""
    seen, todo, stuck = {start}, [start], []
    while todo:
        s = todo.pop()
        nxt = list(successors(s))
        if not nxt:
            stuck.append(s)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return seen, stuck


TILES = 4
ACC, SUM, READ, GONE = range(4)


def _passed(done, n):
    """mbarrier.try_wait on the parity of phase ``n`` when ``done`` phases are complete: it tells neighbouring phases apart only."""
    return (done ^ n) & 1 == 1


def _exchange(bounded):
    """The two epilogue warps of a lane quarter in the convolution with a fused norm. Per tile: wait for the accumulator (bounded: it
    may run out for one warp and not for the other), write the sum of squares into the tile's buffer, meet, read the partner's.
    ``bounded``: they meet at a barrier with a bounded wait (an mbarrier per buffer, two arrivals), else at a named barrier.
    State: tiles finished by the tensor pipe, abort flag, per warp (tile, step), the tile whose sum lies in each warp's two buffers,
    arrivals per warp and buffer."""

    def successors(s):
        ready, abort, warps, bufs, arrived = s
        if ready < TILES:
            yield ready + 1, abort, warps, bufs, arrived
        for i in (0, 1):
            tile, step = warps[i]
            if step == GONE:
                continue
            b = tile & 1

            def to(w, abort=abort, bufs=bufs, arrived=arrived):
                return ready, abort, warps[:i] + (w,) + warps[i + 1:], bufs, arrived

            if step == ACC:
                if ready > tile:                                        # the sum is written and announced
                    nb = tuple(tuple(tile if (j, k) == (i, b) else bufs[j][k] for k in (0, 1)) for j in (0, 1))
                    na = tuple(tuple(arrived[j][k] + ((j, k) == (i, b)) for k in (0, 1)) for j in (0, 1))
                    yield to((tile, SUM), bufs=nb, arrived=na)
                yield to((tile, GONE), abort=1)                          # the limit, or the abort flag, at any moment
            elif step == SUM:
                if bounded:
                    if _passed((arrived[0][b] + arrived[1][b]) // 2, tile >> 1):
                        yield to((tile, READ))
                    yield to((tile, GONE), abort=1)
                elif arrived[1 - i][b] == arrived[i][b] or warps[1 - i][0] > tile:
                    yield to((tile, READ))
            else:
                yield to((tile + 1, ACC) if tile + 1 < TILES else (tile, GONE))

    return (0, 0, ((0, ACC), (0, ACC)), ((-1, -1), (-1, -1)), ((0, 0), (0, 0))), successors


@pytest.mark.parametrize("bounded", [True, False])
def test_exchange_of_sums_between_two_epilogue_warps(bounded):
    seen, stuck = explore(*_exchange(bounded))
    hung = [s for s in stuck if any(w[1] != GONE for w in s[2])]
    if not bounded:
        assert hung, "the model has to show the hang of a named barrier whose partner gave up"
        return
    assert not hung
    for (_, _, warps, bufs, _), i in itertools.product(seen, (0, 1)):
        if warps[i][1] == READ:
            tile = warps[i][0]
            assert bufs[1 - i][tile & 1] == tile, "a warp reads a sum of another tile"


def test_convolution_warps_meet_at_bounded_waits():
    """The convolution kernel is the bounded variant of the model above: no named barrier."""
    assert "bar.sync" not in (CSRC / "conv3d_cl.cu").read_text()


def _meetings(polite):
    """The two element-wise warps of a lane quarter in the single-pass attention backward: per query tile a bounded wait, a meeting at a
    named barrier without a limit, another bounded wait. ``polite``: a warp that gives up leaves a word, which its partner reads at the
    top of every tile, and still arrives at the pair's next meeting; otherwise it just goes. State: the word, per warp (tile, step),
    arrivals per warp."""
    TOP, BEFORE, AT, AFTER, OUT = range(5)

    def successors(s):
        word, warps, came = s
        for i in (0, 1):
            tile, step = warps[i]
            last = tile + 1 == TILES

            def to(step, tile=tile, word=word, arrive=0):
                return (word, warps[:i] + ((tile, step),) + warps[i + 1:], came[:i] + (came[i] + arrive,) + came[i + 1:])

            if step == TOP:
                yield to(OUT if polite and word else BEFORE)
            elif step == BEFORE:
                yield to(AT, arrive=1)
                yield to(OUT, word=1, arrive=int(polite))
            elif step == AT:
                if sum(came) >= 2 * (tile + 1):
                    yield to(AFTER)
            elif step == AFTER:
                yield to(OUT) if last else to(TOP, tile=tile + 1)
                yield to(OUT, word=1, arrive=int(polite and not last))

    return (0, ((0, TOP), (0, TOP)), (0, 0)), successors, OUT


@pytest.mark.parametrize("polite", [True, False])
def test_a_warp_that_gives_up_comes_to_the_next_meeting(polite):
    start, successors, out = _meetings(polite)
    _, stuck = explore(start, successors)
    hung = [s for s in stuck if any(w[1] != out for w in s[1])]
    assert bool(hung) == (not polite)


def test_backward_warps_leave_together():
    """The attention backward is the polite variant: no wait of its element-wise warps just breaks off in front of a meeting."""
    code = (CSRC / "fa_bwd_fused.cu").read_text()
    loop = code[code.index("for (int i = u; i < n_q; i += 2)"):code.index("mbar_wait_warp(done")]
    assert "bar.sync" in loop and "bar.arrive" in code and loop.count("mbar_wait") == 3
    assert loop.count("give_up(") == 2 and "mbar_wait(" not in loop


@pytest.mark.parametrize("path", [p for p in sorted(CSRC.glob("*.cu")) if "tmem_ld" in p.read_text()], ids=lambda p: p.name)
def test_waits_in_front_of_collective_instructions_are_the_warps(path):
    """A wait may run out for some lanes of a warp only. Loads from tensor memory and cluster barriers need every lane, so a warp waits as
    a whole; a plain wait belongs to code that one lane runs."""
    lines = path.read_text().splitlines()
    assert any("mbar_wait" in line for line in lines)
    for n, line in enumerate(lines):
        if "mbar_wait(" not in line or "__all_sync(0xffffffffu, mbar_wait(" in line:
            continue
        depth = len(line) - len(line.lstrip())
        for above in reversed(lines[:n]):                       # the statement that opens the nearest enclosing role
            d = len(above) - len(above.lstrip())
            if above.strip() and above[0] != "#" and d < depth:
                depth = d
                if "lane == 0" in above or "else if (warp" in above or "} else {" in above:
                    break
        assert "if (lane == 0) {" in above, f"{path.name}:{n + 1} waits lane by lane"


def _early_kernels():
    """(name, parameters, body up to the wait) of every kernel that may start beside the kernel in front of it."""
    for path in sorted(CSRC.glob("*.cu")):
        for part in re.split(r"\n__global__ ", path.read_text())[1:]:
            part = part.split("\n}\n")[0]
            if "pdl_wait();" in part:
                head, body = part.split(") {\n", 1)
                name, params = re.search(r"(\w+_kernel)\((.*)$", head, re.S).groups()
                yield name, params, body[:body.rindex("pdl_wait();")]


_VALUES = {"int", "long", "float", "bool", "unsigned", "uint8_t", "int8_t", "uint32_t", "int32_t", "int64_t", "uint64_t", "size_t", "CUtensorMap"}


def _struct(name, code):
    """Members of a struct: (name, type, whether a pointer, whether an array)."""
    body = re.search(rf"\bstruct (?:alignas\(\d+\) )?{name} {{(.*?)\n}};", code, re.S)
    assert body, f"no definition of {name}: its pointers cannot be looked for"
    members = []
    for decl in re.sub(r"//[^\n]*", "", body.group(1)).split(";"):
        decl = " ".join(decl.split())
        if not decl or "(" in decl and "[" not in decl:
            continue
        m = re.match(r"(?:const |static |constexpr )*([\w:]+(?: long)?(?:<\w+>)?)\s*(.*)$", decl)
        for part in m.group(2).split(","):
            d = re.match(r"\s*(?:const )?(\**)\s*(?:const |__restrict__ )*(\**)\s*(\w+)\s*((?:\[[^\]]*\])*)", part)
            assert d, f"{name}: cannot read the member {decl!r}"
            members.append((d.group(3), m.group(1).split("<")[0], bool(d.group(1) or d.group(2)), bool(d.group(4))))
    return members


def _pointers(type_, path, code):
    """Patterns of the expressions that are pointers inside a by-value parameter."""
    for name, t, pointer, array in _struct(type_, code):
        at = rf"{path}\.{name}" + (r"\s*\[[^\]]*\]" if array else "")
        if pointer:
            yield at
        elif t not in _VALUES:
            yield from _pointers(t, at, code)


def _reads_ahead(params, ahead, code):
    """The first access, ahead of the wait, to memory that a parameter points to; the device's error word is open, tensor maps are no such
    memory."""
    pointers = []
    for p in re.split(r",(?![^<]*>)", params):
        type_, var = re.match(r"\s*(.*?)(\w+)\s*$", " ".join(p.split())).groups()
        base = re.sub(r"\b(const|volatile|__grid_constant__|__restrict__)\b|<\w+>|[*&]", "", type_).strip()
        if var == "err":
            continue
        if "*" in type_:
            pointers.append(rf"\b{var}")
        elif base not in _VALUES:
            pointers += list(_pointers(base, rf"\b{var}", code))
    # what is set to such a pointer (or to it with an offset) is one as well
    for _ in range(3):
        for ptr in list(pointers):
            for name in re.findall(rf"\b(\w+) = (?:reinterpret_cast<[^>]*>\()?\(?{ptr}\)?(?: \+ [^;]*)?;", ahead):
                if rf"\b{name}" not in pointers:
                    pointers.append(rf"\b{name}")
    for ptr in pointers:
        # (a pointer behind a star is read, unless it is declared there: pointers are not multiplied)
        hit = re.search(rf"{ptr}\s*\[|\*\s*\(?{ptr}(?!\w)(?! =[^=])|\({ptr}\s*\+|reinterpret_cast<[^>]*>\({ptr}\)\s*\[", ahead)
        if hit:
            return hit.group(0)
    hit = re.search(r"\b(?:tma_load\w*|bulk_load\w*|tma_store\w*|atomic\w+|red_\w+)\(", ahead)
    return hit and hit.group(0)


def test_kernels_read_no_memory_ahead_of_their_wait():
    """What the kernel in front writes is visible behind ``pdl_wait()`` only. Ahead of it a kernel touches no memory that its parameters
    point to, except the device's error word; hints that bring a tile into L2 read nothing."""
    code = "\n".join(p.read_text() for p in sorted([*CSRC.glob("*.cuh"), *CSRC.glob("*.h"), *CSRC.glob("*.cu")]))
    kernels = list(_early_kernels())
    assert len(kernels) >= 12
    for name, params, ahead in kernels:
        hit = _reads_ahead(params, ahead, code)
        assert hit is None, f"{name} reads ahead of the wait: {hit}"


def test_reads_ahead_of_a_wait_are_found():
    """Plain pointers, members of by-value structs whatever the parameter's name, arrays of pointers, nested structs, what is set to them."""
    code = """
struct Inner {
  float* sums[8];   // one a rank
  int n;
};
struct Outer {
  const bf16 *a, *b;
  void* out[NW];
  CUtensorMap map[3];
  Inner in;
  long ld;
};
"""
    outer = "const __grid_constant__ Outer things, const float* __restrict__ x, int n, int* err"
    for bad in ("v = things.a[i];", "v = *things.b;", "things.out[g][i] = 0;", "f(*things.in.sums[r]);", "g(things.a + 4);", "v = x[0];", "const bf16* q = things.a; v = q[2];",
                "tma_load_2d(s, &m, bar, 0, 0);", "v = reinterpret_cast<const float4*>(x)[i];"):
        assert _reads_ahead(outer, bad, code), bad
    for good in ("prefetch_tmap(&things.map[g]);", "tma_prefetch_l2_2d(&things.map[0], 0, n);", "bool has = things.a != nullptr;", "int k = things.in.n * n;",
                 "const bf16* q = things.a;", "if (*err) return;", "long m = things.ld * n;"):
        assert _reads_ahead(outer, good, code) is None, good
    with pytest.raises(AssertionError):
        _reads_ahead("Unknown u", "", code)


_SIZES = {"char": 1, "uint8_t": 1, "int8_t": 1, "bf16": 2, "__nv_bfloat16": 2, "half": 2, "float": 4, "int": 4, "uint32_t": 4, "int32_t": 4,
          "__nv_bfloat162": 4, "float2": 8, "uint2": 8, "int2": 8, "long": 8, "double": 8, "int64_t": 8, "uint64_t": 8, "float4": 16, "uint4": 16,
          "int4": 16, "bf16x8": 16}


def _wider_accesses(code):
    """(line, array, its type, type it is accessed as) where a cast reads an array as a type that asks for more alignment than the array has."""
    for cast in re.finditer(r"reinterpret_cast<(?:const )?(\w+)\*>\(&?(\w+)(?:\[[^\]]*\])?\)", code):
        wide, var = cast.groups()
        found = [d for d in re.finditer(rf"^[ \t]*([^\n;(){{}}]*?\b)(\w+) {var}(?:\[[^\]]*\])+ *(?=[=;,{{])", code, re.M) if d.start() < cast.start()]
        if not found or wide not in _SIZES or found[-1].group(2) not in _SIZES:
            continue
        qualifiers, narrow = found[-1].groups()
        if _SIZES[wide] > _SIZES[narrow] and "align" not in qualifiers and "align" not in found[-1].group(0):
            yield code[:cast.start()].count("\n") + 1, var, narrow, wide


def test_arrays_are_aligned_for_the_accesses_to_them():
    """An array that is read or written through a wider type is declared with that type's alignment: in local memory the access faults."""
    assert list(_wider_accesses("  bf16 e[8];\n  x = *reinterpret_cast<const bf16x8*>(e);\n")) == [(2, "e", "bf16", "bf16x8")]
    assert not list(_wider_accesses("  alignas(16) bf16 e[8];\n  x = *reinterpret_cast<const bf16x8*>(e);\n"))
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        assert list(_wider_accesses(path.read_text())) == [], path.name
