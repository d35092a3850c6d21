"""Which launches run beside each other (LcOrder and LcPlain, csrc/abi.cu, csrc/lc_internal.h), without a GPU: a host program makes the
decisions for random sequences of launches, and a model of the stream checks that no launch touches what one that may still be
running writes, or writes what one may still be reading."""
import random
import subprocess

import pytest

PROGRAM = r'''
#include "abi.cu"
void lc_cluster_capacity(const lc_ctx *, uint32_t (&)[9]) {}
int main() {
    lc_ctx ctx;
    ctx.stream = (cudaStream_t)0x10;
    lc_batch b;
    b.ctx = &ctx;
    b.stream = ctx.stream;
    char kind;
    while (scanf(" %c", &kind) == 1) {
        uint32_t flags = 0, serial = 0;
        if (kind == 'm') {
            size_t at[3];
            int brief;
            lc_buf bufs[3];
            if (scanf("%zu %zu %zu %d", &at[0], &at[1], &at[2], &brief) != 4) return 1;
            for (int i = 0; i < 3; i++) bufs[i].dptr = (void *)(at[i] * 16 + 4096);
            const lc_buf *w = &bufs[1];
            lc_buf *out = &bufs[2];
            const size_t n = 16;
            LcOrder o(&b, &bufs[0], n, 1, &w, &n, &out, &n, brief);
            flags = o.flags;
            serial = o.serial;
            o.launched = true;
        } else if (kind == 'p') {
            LcPlain p(&b);
            serial = p.serial;
        } else {
            lc_order_break(&ctx, kind == 'f');
        }
        printf("%u %u\n", flags, serial);
    }
}
'''


@pytest.fixture(scope="module")
def decide(la, tmp_path_factory):
    import importlib
    build = importlib.import_module("__graft_entry__").load_build_module()
    at = tmp_path_factory.mktemp("order")
    (at / "order.cu").write_text(PROGRAM)
    subprocess.run([build.find_nvcc(), "-std=c++17", f"-I{build.CSRC}", str(at / "order.cu"), "-o", str(at / "order")], check=True, capture_output=True)

    def run(ops):
        text = "\n".join(" ".join(map(str, op)) for op in ops)
        out = subprocess.run([str(at / "order")], input=text, check=True, capture_output=True, text=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return run


def conflicts(ops, orders):
    """Pairs (i, j): launch i works on data of launch j, which need not be complete then.  Everything before launch `done[i]` is complete when
    launch i works on its data, before `trig[i]` when its successor may start and before `end[i]` when it is complete itself."""
    bad, trig, end = [], 0, 0
    for i, (op, (flags, serial)) in enumerate(zip(ops, orders)):
        start = max(trig, i if serial else 0) if op[0] in "mp" else i
        if op[0] == "m" and flags == 2:
            data, trig, end = start, start, i
        elif op[0] == "m" and flags == 1:
            data, trig, end = i, i, i
        elif op[0] == "c":
            data, trig, end = i, i + 1, i
        elif op[0] == "f":                       # (may let its successor start early)
            data, trig, end = i, i, i
        else:
            data, trig, end = i, start, i
        if op[0] == "m":
            for j in range(data, i):
                if ops[j][0] in "pf" or ops[j][3] in op[1:3] or op[3] in ops[j][1:4]:
                    bad.append((i, j))
    return bad


def matmul(rng, spots):
    return ("m", rng.randrange(spots), 1000 + rng.randrange(3), rng.randrange(spots), int(rng.random() < 0.3))


@pytest.mark.parametrize("spots", [4, 12, 400])
def test_nothing_meets(decide, spots):
    rng = random.Random(spots)
    beside = 0
    for _ in range(20):
        ops = [matmul(rng, spots) if rng.random() < 0.85 else (rng.choice("pcf"),) for _ in range(300)]
        orders = decide(ops)
        assert not conflicts(ops, orders)
        beside += sum(flags == 2 for flags, _ in orders)
    assert beside


def test_other_work_ends_a_run(decide):
    run = [("m", 1, 1000, 10 + i, 0) for i in range(4)]
    for kind in "pcf":
        orders = decide(run + [(kind,)] + run)
        assert [f for f, _ in orders] == [0, 1, 2, 2, 0, 0, 1, 2, 2]
        # a launch behind a run starts when the run is complete, also where another library's kernel stands between
        assert orders[4 if kind == "p" else 5][1] == (kind != "c")


def test_a_full_list(decide):
    """The lists hold 96 writes.  A launch that finds them full and meets the run starts when the run is complete, since the next one
    knows only of it."""
    ops = [("m", 1, 1000, 10 + i, 0) for i in range(97)]
    ops += [("m", 50, 1000, 200, 0), ("m", 1, 60, 300, 0)]
    orders = decide(ops)
    assert [f for f, _ in orders][:97] == [0] + [1] + [2] * 95
    assert not conflicts(ops, orders) and orders[97] == (0, 1)


def test_brief_launches_start_no_run(decide):
    """Two launches that the host enqueues more slowly than the GPU runs them stay one behind the other; beside a longer one they do not."""
    run = [("m", 1, 1000, 10 + i, 1) for i in range(4)]
    assert decide(run) == [(0, 0)] * 4
    assert [f for f, _ in decide([("m", 1, 1000, 9, 0)] + run)] == [0, 1, 2, 2, 2]
    assert [f for f, _ in decide(run + [("m", 1, 1000, 9, 0)] + run[:2])] == [0, 0, 0, 0, 1, 2, 2]
