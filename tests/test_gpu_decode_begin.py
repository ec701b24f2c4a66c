"""A decode step's first launches: tokens, slots, positions and lengths in one, the embedding's rows with their sums of squares."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("advance", [True, False])
@pytest.mark.parametrize("n,slots", [(1, 1), (8, 9), (64, 70), (129, 300)])
def test_decode_begin(n, slots, advance):
    """Every sequence's token, slot and position; its length goes up by one, or stays for the launch behind the step."""
    from dryft_b200.ops import kernels as K

    gen = torch.Generator().manual_seed(n)
    seq_slot = torch.randperm(slots, generator=gen)[:n]
    seq_slot[n // 2::3] = -1                                # padding rows
    last, lens = torch.randint(0, 1000, (slots,), generator=gen), torch.randint(0, 5000, (slots,), generator=gen)
    live = seq_slot >= 0
    want = [torch.where(live, last[seq_slot], 0), seq_slot, torch.where(live, lens[seq_slot], 0)]
    after = lens.clone()
    after[seq_slot[live]] += 1
    i32 = lambda t: t.to(torch.int32).cuda()
    d_slot, d_lens = i32(seq_slot), i32(lens)
    got = [torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(3)]
    K.decode_begin(d_slot, i32(last), d_lens, got[0], got[1], got[2], n, advance=advance)
    assert all(torch.equal(a, i32(b)) for a, b in zip(got, want))
    if not advance:
        assert torch.equal(d_lens, i32(lens))
        K.step_advance(torch.arange(n + 1, dtype=torch.int32, device="cuda"), d_slot, d_lens, n)
    assert torch.equal(d_lens, i32(after))


@pytest.mark.parametrize("n,hidden", [(1, 1024), (16, 2560), (64, 80), (3, 37)])
def test_embedding_rows_with_their_sums_of_squares(n, hidden):
    from dryft_b200.ops import kernels as K

    table = torch.randn(50, hidden, device="cuda").bfloat16()
    toks = torch.randint(0, 50, (n,), device="cuda").to(torch.int32)
    toks[n // 2] = 50 if n > 1 else toks[0]                  # outside the table: a row of zeros
    rows, ss, err = torch.empty(n, hidden, dtype=torch.bfloat16, device="cuda"), torch.full((64,), -1.0, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    K.embed(toks, table, rows, err, ss)
    plain, ss2 = torch.empty_like(rows), torch.empty(64, device="cuda")
    K.embed(toks, table, plain)
    K.row_sumsq(plain, ss2)
    assert torch.equal(rows, plain) and torch.equal(ss[:n], ss2[:n]) and int(err) == (1 if n > 1 else 0)


@pytest.mark.parametrize("graphs", [False, True])
def test_a_step_that_raises_leaves_the_lengths_as_they_were(model_dirs, graphs):
    """An eager decode step that ends in an error half-way has appended nothing: device and host agree on the lengths, and the
    step done again gives the logits of one that was never disturbed.  (A captured step is replayed whole or not at all.)"""
    from dryft_b200.engine.api import Engine

    def run(disturb):
        eng = Engine(model_dirs["a"], dtype="bfloat16", max_batch=4, max_seq_len=256, max_tokens=1024, cuda_graphs=graphs)
        out = []
        with torch.inference_mode():
            slots = eng.cache.open_sequences(3)
            eng.stepper.step(slots, [[1, 2, 3], [4] * 20, [5]], [[], [], []])
            at = torch.tensor(slots, device="cuda")
            for t in range(4):
                eng.cache.last_token.index_copy_(0, at, torch.tensor([t + 1, 2 * t, 3], dtype=torch.int32, device="cuda"))
                if disturb and t in (0, 2):
                    forward = eng.model.forward
                    if graphs and t == 2:
                        eng.stepper._graphs.clear()          # another capture, which fails
                    eng.model.forward = lambda *a, **k: (forward(*a, **k), 1 / 0)
                    with pytest.raises(ZeroDivisionError):
                        eng.stepper.decode_from_state(slots)
                    del eng.model.forward
                    torch.cuda.synchronize()
                    assert [int(n) for n in eng.cache.seq_len[at]] == [eng.cache.len_host[s] for s in slots]
                out.append(eng.stepper.decode_from_state(slots)[:3].clone())
            assert [int(n) for n in eng.cache.seq_len[at]] == [eng.cache.len_host[s] for s in slots]
        return torch.stack(out)

    assert torch.equal(run(True), run(False))
