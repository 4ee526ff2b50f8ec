"""Delimited text parsed from shared-memory copies: fields around the short
reader's eight bytes, records that fit the copy and records that do not,
string bytes at every output alignment and at the file's last bytes."""
import numpy as np
import pytest
import torch

import oracle_bind as ob
from test_csv_gpu import assert_same

pytestmark = pytest.mark.gpu

NUMBERS = ["0", "-0", "0.0", "-.5", ".5", "5.", "-", ".", "-.", "", "1.2.3", "12345678", "1234567.", "1234567.8",
           "12345.67", "-123.456", "-1234.567", "99999999", "123456789", "1e5", "12e-3", "1.5E2", "007", "-00.10",
           "+1", "1x", "x1", "1 2", "nan", "-inf", "4294967295", "4294967296", "0.1234567", "0.12345678", "9999999.9"]
STRINGS = ["", "a", "bc", "def", "ghij", "klmno", "\"p,q\"", "NA", "a much longer string of text, quoted".replace(",", ""),
           "\"x\ny\"", "0123456789abcdef"]


def check(ctx, text):
    data = text.encode()
    t = ctx.read_csv(torch.from_numpy(np.frombuffer(data, dtype=np.uint8).copy()).cuda(), quote='"')
    assert_same(t, ob.csv_read(data, quote='"'))
    t.close()


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 128, 255, 257, 5000])
@pytest.mark.parametrize("eol", ["\n", "\r\n"])
@pytest.mark.parametrize("end", [True, False])
def test_fields(ctx, rows, eol, end):
    rng = np.random.default_rng(rows)
    lines = ["d,u,b,s,z"]
    for r in range(rows):
        first = r < 10  # the first rows decide the types
        num = "1.5" if first else NUMBERS[rng.integers(len(NUMBERS))]
        u = "12" if first else NUMBERS[rng.integers(len(NUMBERS))]
        b = "1" if first else NUMBERS[rng.integers(len(NUMBERS))]
        lines.append(",".join([num, u, b, STRINGS[rng.integers(len(STRINGS))] if not first else "text",
                               STRINGS[rng.integers(len(STRINGS))] if not first else "more"]))
    check(ctx, eol.join(lines) + (eol if end else ""))


@pytest.mark.parametrize("long", [100, 900, 1100, 3000])
def test_records_longer_than_the_copy(ctx, long):
    """Some CTAs' records exceed the shared copy, others' do not."""
    rng = np.random.default_rng(long)
    lines = ["d,s"]
    for r in range(700):
        k = int(rng.integers(0, long)) if 200 < r < 300 else 3
        lines.append(f"{r}.25," + "abcdefghij"[r % 10] * (k + (r < 10) * 2))
    check(ctx, "\n".join(lines) + "\n")


def test_many_columns(ctx):
    rng = np.random.default_rng(7)
    for ncol in (63, 64, 65, 1500):
        rows = [",".join(f"c{k}" for k in range(ncol))]
        rows += [",".join(f"{x:.2f}" for x in rng.random(ncol) * 100) for _ in range(40)]
        check(ctx, "\n".join(rows) + "\n")


def test_sixty_four_string_columns(ctx):
    rows = [",".join(f"c{k}" for k in range(64))]
    rows += [",".join("abcdefgh"[: 2 + (r + k) % 7] for k in range(64)) for r in range(70)]
    check(ctx, "\n".join(rows) + "\n")
