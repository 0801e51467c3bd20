"""ctypes mirrors of the structs in include/tha_hybrid.h that the tests of single mechanisms fill in themselves."""
import ctypes as C

from pkgload import load_pkg

I, F, P, L = C.c_int, C.c_float, C.c_void_p, C.c_longlong


def _struct(name, fields):
    return type(name, (C.Structure,), {"_fields_": [(n, t) for names, t in fields for n in names.split()]})


Rows = _struct("tha_rows_t", [("n_rows n_seqs", I), ("token pos row_seq seq_first seq_slot", P), ("max_seq_rows max_pos", I)])
Kv = _struct("tha_kv_t", [("k_pool v_pool table", P), ("table_stride block_size n_cache_layers kv_dim", I)])
States = _struct("tha_state_store_t", [("base", P), ("slot_floats", L)])
Norm = _struct("tha_norm_t", [("kind", I), ("w b", P), ("w_offset alpha", F)])
Attn = _struct("tha_attn_t", [("heads kv_heads dim vdim rot unit_rms", I), ("eps scale", F), ("chunk cache_layer o_q o_k o_v", I), ("w_o", P),
                              ("values_in_keys window keep_first", I), ("sink head_scale", P), ("rot_layout head_gate o_g fp32_scores v_share out_f32", I),
                              ("q_temp_coef", F), ("q_temp_every kv_shared diff", I), ("diff_lambda diff_mult", F), ("conv_taps", I), ("conv_w", P),
                              ("conv_state_off", L), ("conv_b", P), ("v_is_k", I), ("q_norm k_norm", P), ("softcap", F), ("b_o", P), ("head_norm", I),
                              ("rel", P), ("rel_n v_mix v_mix_layer", I), ("v_mix_lambda", F)])
Model = _struct("tha_hyb_model_t", [("dtype width vocab n_layers", I), ("eps logit_softcap", F), ("embed pos_embed", P), ("max_positions", I), ("final_norm", Norm),
                                    ("head layers", P), ("n_rot", I), ("rot", P), ("embed_scale", F), ("side_table", P), ("side_cols n_streams", I)])
STRUCTS = (Rows, Kv, States, Norm, Attn, Model)
BF16, F32 = 0, 1


def ptr(t):
    return t.data_ptr() if t is not None else None


def lib():
    """The library with the argument types of the calls that these tests make."""
    lib = load_pkg("cabi").lib()
    c = lib.c
    c.tha_hyb_step.argtypes = [P, C.POINTER(Model), C.POINTER(Rows), C.POINTER(Kv), C.POINTER(States), I, P, P, P]
    c.tha_hyb_rmsnorm.argtypes = [P, I, P, P, P, F, F, I, I, P]
    c.tha_hyb_attn.argtypes = [P, I, C.POINTER(Attn), C.POINTER(Rows), C.POINTER(Kv), P, P, P, C.c_size_t]
    return lib


def rows_of(seqs, block=64):
    """seqs: [(slot, first position, rows)] -> (Rows, what keeps its device arrays alive)."""
    import numpy as np
    import torch
    pos = np.concatenate([p0 + np.arange(n) for _, p0, n in seqs])
    seq = np.concatenate([np.full(n, i) for i, (_, _, n) in enumerate(seqs)])
    first = np.cumsum([0] + [n for _, _, n in seqs])
    arrays = [torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda() for a in (np.zeros_like(pos), pos, seq, first, np.array([s for s, _, _ in seqs]))]
    return Rows(len(pos), len(seqs), *[a.data_ptr() for a in arrays], max(n for _, _, n in seqs), int(pos.max())), arrays
