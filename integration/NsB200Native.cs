// GENERATED by integration/gen_native_cs.py from include/ns_b200.h -- do not edit by hand.
// NOT COMPILED: no .NET SDK exists where this library is built; tests/test_integration_cs.py checks every import
// against the header (name, parameter count, integer widths).
//
// Sibling of src/NeuralSharp/Backends/Cuda/CudaDriver.cs: the same resolver and Check conventions, one import per
// function of the C ABI.  Device addresses are ulong (CUdeviceptr in the reference), handles are nint.
using System.Reflection;
using System.Runtime.InteropServices;

namespace NeuralSharp.Backends.B200;

/// <summary>Thrown when a libns_b200 call returns a non-zero code.</summary>
public sealed class NsB200Exception(string message, int code) : Exception(message)
{
    public int Code { get; } = code;
}

internal static unsafe partial class NsB200Native
{
    private const string Library = "ns_b200";

    public const int Ok = 0, ErrCuda = 1, ErrArgument = 2, ErrMemory = 3, ErrKernel = 4, ErrComm = 5, ErrState = 6;
    public const int F32 = 0, Bf16 = 1, I8 = 2, I32 = 3;
    public const int EpiNone = 0, EpiBias = 1, EpiBiasGelu = 2, EpiBiasResidual = 3;
    public const int SplitNone = 0, SplitColumn = 1, SplitRow = 2;

    static NsB200Native()
    {
        NativeLibrary.SetDllImportResolver(typeof(NsB200Native).Assembly, Resolve);
    }

    /// <summary>True when libns_b200.so can be loaded (it opens only devices of compute capability 10.x).</summary>
    public static bool TryLoad(out string reason)
    {
        foreach (var name in CandidateNames())
        {
            if (NativeLibrary.TryLoad(name, out var handle))
            {
                NativeLibrary.Free(handle);
                reason = "";
                return true;
            }
        }

        reason = $"libns_b200 ({string.Join(" / ", CandidateNames())}) was not found";
        return false;
    }

    private static IntPtr Resolve(string name, Assembly assembly, DllImportSearchPath? searchPath)
    {
        if (name != Library)
        {
            return IntPtr.Zero;
        }

        foreach (var candidate in CandidateNames())
        {
            if (NativeLibrary.TryLoad(candidate, assembly, searchPath, out var handle))
            {
                return handle;
            }
        }

        return IntPtr.Zero;
    }

    private static string[] CandidateNames() =>
        Environment.GetEnvironmentVariable("NS_B200_LIBRARY") is { Length: > 0 } path ? [path, "libns_b200.so"] : ["libns_b200.so"];

    /// <summary>Turns a non-zero return code into an exception carrying the library's text for the calling thread.</summary>
    public static void Check(int result, string call)
    {
        if (result == 0)
        {
            return;
        }

        string text = Marshal.PtrToStringUTF8(ns_last_error()) ?? "";
        string name = Marshal.PtrToStringUTF8(ns_error_name(result)) ?? "NS_ERR_UNKNOWN";
        throw new NsB200Exception($"{call} failed: {text} ({name}, {result})", result);
    }

    [LibraryImport(Library)]
    public static partial nint ns_last_error();

    [LibraryImport(Library)]
    public static partial nint ns_error_name(int code);

    [LibraryImport(Library)]
    public static partial int ns_version();

    [LibraryImport(Library)]
    public static partial int ns_device_count(out int count);

    [LibraryImport(Library)]
    public static partial int ns_device_open(int ordinal, out nint dev);

    [LibraryImport(Library)]
    public static partial int ns_device_open_on_stream(int ordinal, ulong stream, out nint dev);

    [LibraryImport(Library)]
    public static partial int ns_device_close(nint dev);

    [LibraryImport(Library)]
    public static partial int ns_device_info(nint dev, byte* name, int* sm_count, ulong* total_bytes, ulong* free_bytes);

    [LibraryImport(Library)]
    public static partial int ns_device_stream(nint dev, out ulong stream);

    [LibraryImport(Library)]
    public static partial int ns_stream_sync(nint dev);

    [LibraryImport(Library)]
    public static partial int ns_device_status(nint dev, out int status);

    [LibraryImport(Library)]
    public static partial int ns_debug_tail_times(nint dev, ulong buffer);

    [LibraryImport(Library)]
    public static partial int ns_device_tune(nint dev, int tile_n, int k_splits);

    [LibraryImport(Library)]
    public static partial int ns_alloc(nint dev, ulong bytes, int zeroed, out ulong ptr);

    [LibraryImport(Library)]
    public static partial int ns_free(nint dev, ulong ptr);

    [LibraryImport(Library)]
    public static partial int ns_h2d(nint dev, ulong dst, void* src, ulong bytes);

    [LibraryImport(Library)]
    public static partial int ns_d2h(nint dev, void* dst, ulong src, ulong bytes);

    [LibraryImport(Library)]
    public static partial int ns_h2d_async(nint dev, ulong dst, void* src, ulong bytes);

    [LibraryImport(Library)]
    public static partial int ns_d2h_async(nint dev, void* dst, ulong src, ulong bytes);

    [LibraryImport(Library)]
    public static partial int ns_d2d_async(nint dev, ulong dst, ulong src, ulong bytes);

    [LibraryImport(Library)]
    public static partial int ns_d2d_2d_async(nint dev, ulong dst, ulong dst_pitch, ulong src, ulong src_pitch, ulong width_bytes, ulong rows);

    [LibraryImport(Library)]
    public static partial int ns_memset32_async(nint dev, ulong dst, uint value, ulong count);

    [LibraryImport(Library)]
    public static partial int ns_host_alloc(ulong bytes, out nint ptr);

    [LibraryImport(Library)]
    public static partial int ns_host_free(void* ptr);

    [LibraryImport(Library)]
    public static partial int ns_ipc_handle(nint dev, ulong ptr, void* handle64);

    [LibraryImport(Library)]
    public static partial int ns_ipc_open(nint dev, void* handle64, out ulong ptr);

    [LibraryImport(Library)]
    public static partial int ns_ipc_close(nint dev, ulong ptr);

    [LibraryImport(Library)]
    public static partial int ns_capture_begin(nint dev);

    [LibraryImport(Library)]
    public static partial int ns_capture_end(nint dev, out nint graph);

    [LibraryImport(Library)]
    public static partial int ns_capture_abort(nint dev);

    [LibraryImport(Library)]
    public static partial int ns_graph_launch(nint dev, nint graph);

    [LibraryImport(Library)]
    public static partial int ns_graph_destroy(nint graph);

    [LibraryImport(Library)]
    public static partial int ns_event_create(nint dev, out ulong @event);

    [LibraryImport(Library)]
    public static partial int ns_event_record(nint dev, ulong @event);

    [LibraryImport(Library)]
    public static partial int ns_event_elapsed_ms(nint dev, ulong start, ulong stop, out float ms);

    [LibraryImport(Library)]
    public static partial int ns_stream_wait_event(nint dev, ulong @event);

    [LibraryImport(Library)]
    public static partial int ns_event_destroy(nint dev, ulong @event);

    [LibraryImport(Library)]
    public static partial int ns_quantize_rows_i8(nint dev, ulong x, int in_dtype, long rows, int cols, ulong q, ulong scale);

    [LibraryImport(Library)]
    public static partial int ns_qmatmul_i8(nint dev, ulong aq, ulong a_scale, ulong wq, ulong w_scale, ulong bias, ulong residual, int residual_dtype, int M, int N, int K, int epilogue, int out_dtype, ulong y, ulong raw_s32);

    [LibraryImport(Library)]
    public static partial int ns_qmatmul_i8_static(nint dev, ulong aq, ulong a_scale, ulong wq, ulong w_scale, ulong bias, ulong residual, int residual_dtype, int M, int N, int K, int epilogue, int out_dtype, ulong y);

    [LibraryImport(Library)]
    public static partial int ns_bench_i8_mainloop(nint dev, ulong aq, ulong wq, int M, int N, int K);

    [LibraryImport(Library)]
    public static partial int ns_matmul_bf16(nint dev, ulong a, ulong b, ulong c, int batch, int m, int n, int k, int transB, ulong bias, ulong residual, int residual_dtype, int epilogue, int out_dtype);

    [LibraryImport(Library)]
    public static partial int ns_layernorm(nint dev, ulong x, int in_dtype, ulong gamma, ulong beta, long rows, int cols, float eps, int out_dtype, ulong y, ulong y_scale);

    [LibraryImport(Library)]
    public static partial int ns_embed_pos(nint dev, ulong ids, ulong tok_table, ulong pos_table, int table_dtype, ulong pos_dev, int batch, int steps, int dim, int vocab, int max_pos, int out_dtype, ulong y);

    [LibraryImport(Library)]
    public static partial int ns_argmax_i32(nint dev, ulong x, int rows, int cols, long row_stride, ulong ids);

    [LibraryImport(Library)]
    public static partial int ns_add_i32(nint dev, ulong counter, int delta);

    [LibraryImport(Library)]
    public static partial int ns_convert(nint dev, ulong x, int in_dtype, ulong y, int out_dtype, long n);

    [LibraryImport(Library)]
    public static partial int ns_fill_normal(nint dev, ulong y, int dtype, long n, uint seed, float mean, float std);

    [LibraryImport(Library)]
    public static partial int ns_fill_ids(nint dev, ulong y, long n, uint seed, uint bound);

    [LibraryImport(Library)]
    public static partial int ns_f32_batched_matmul(nint dev, ulong a, ulong b, ulong c, int batch, int m, int n, int k, int transA, int transB, float beta);

    [LibraryImport(Library)]
    public static partial int ns_f32_scale_mask_softmax(nint dev, ulong x, ulong mask, ulong y, int rows, int cols, int maskRows, float scale);

    [LibraryImport(Library)]
    public static partial int ns_f32_layernorm_fused(nint dev, ulong x, ulong gamma, ulong beta, ulong y, int rows, int cols, float eps);

    [LibraryImport(Library)]
    public static partial int ns_f32_bias_gelu(nint dev, ulong x, ulong bias, ulong y, long n, int cols);

    [LibraryImport(Library)]
    public static partial int ns_f32_add_row_vector(nint dev, ulong a, ulong v, ulong c, int rows, int cols);

    [LibraryImport(Library)]
    public static partial int ns_f32_add(nint dev, ulong a, ulong b, ulong c, long n);

    [LibraryImport(Library)]
    public static partial int ns_f32_affine(nint dev, ulong x, ulong y, long n, float alpha, float beta);

    [LibraryImport(Library)]
    public static partial int ns_f32_add_broadcast_scalar(nint dev, ulong s, ulong y, long n, float scale);

    [LibraryImport(Library)]
    public static partial int ns_f32_decoder_mask(nint dev, ulong position, ulong mask, int rows, int capacity);

    [LibraryImport(Library)]
    public static partial int ns_f32_key_value_write(nint dev, ulong source, ulong cache, ulong position, int heads, int steps, int capacity, int dim);

    [LibraryImport(Library)]
    public static partial int ns_f32_gather(nint dev, ulong table, ulong indices, ulong y, int count, int dim, int vocabulary);

    [LibraryImport(Library)]
    public static partial int ns_f32_argmax(nint dev, ulong x, ulong y, int rows, int cols);

    [LibraryImport(Library)]
    public static partial int ns_f32_argmax_strided(nint dev, ulong x, ulong y, int rows, int cols, long row_stride, long row_offset);

    [LibraryImport(Library)]
    public static partial int ns_f32_permute(nint dev, ulong x, ulong y, int* outShape, int* inStrides, int rank, int accumulate);

    [LibraryImport(Library)]
    public static partial int ns_f32_copy2d(nint dev, ulong src, long srcOffset, int srcStride, ulong dst, long dstOffset, int dstStride, int rows, int cols, int accumulate);

    [LibraryImport(Library)]
    public static partial int ns_f32_linear(nint dev, ulong x, ulong gamma, ulong beta, float eps, ulong w, ulong bias, ulong residual, int gelu, ulong y, int m, int n, int k);

    [LibraryImport(Library)]
    public static partial int ns_f32_attention_step(nint dev, ulong qkv, ulong keys, ulong values, ulong position, ulong y, int batch, int heads, int capacity, int dim, float scale);

    [LibraryImport(Library)]
    public static partial int ns_f32_embed_positions(nint dev, ulong ids, ulong table, ulong positions, ulong position, ulong x, int batch, int steps, int dim, int vocabulary, int capacity);

    [LibraryImport(Library)]
    public static partial int ns_f32_sample_rows(nint dev, ulong logits, ulong ids, ulong stats, ulong step, int rows, int vocabulary, int rowStride, int rowOffset, float temperature, int topK, float topP, float minP, uint seed);

    [LibraryImport(Library)]
    public static partial int ns_f32_penalize_rows(nint dev, ulong logits, ulong work, ulong history, ulong length, int rows, int vocabulary, int rowStride, int rowOffset, int capacity, int lastN, float repeat, float presence, float frequency);

    [LibraryImport(Library)]
    public static partial int ns_f32_history_push(nint dev, ulong ids, ulong history, ulong length, int rows, int capacity);

    [LibraryImport(Library)]
    public static partial int ns_kv_cache_create(nint dev, int num_pages, int page_size, int heads, int head_dim, out nint cache);

    [LibraryImport(Library)]
    public static partial int ns_kv_cache_create_in(nint dev, int num_pages, int page_size, int heads, int head_dim, ulong k_pool, ulong v_pool, out nint cache);

    [LibraryImport(Library)]
    public static partial int ns_kv_cache_destroy(nint cache);

    [LibraryImport(Library)]
    public static partial int ns_kv_scatter_heads(nint dev, nint src, ulong src_table, int src_max_pages, int n_seqs, int seq0, int pages_used, ulong* dst_k_pools, ulong* dst_v_pools, int world, int dst_heads, int dst_num_pages, ulong dst_table, int dst_max_pages, int layers, ulong src_layer_stride, ulong dst_layer_stride);

    [LibraryImport(Library)]
    public static partial int ns_kv_cache_pools(nint cache, ulong* k_pool, ulong* v_pool, ulong* bytes_each);

    [LibraryImport(Library)]
    public static partial int ns_kv_append(nint dev, nint cache, ulong k, ulong v, long src_stride, ulong page_table, int max_pages, ulong pos_dev, int batch, int steps);

    [LibraryImport(Library)]
    public static partial int ns_attention_decode(nint dev, nint cache, ulong q, long q_stride, ulong o, long o_stride, ulong page_table, int max_pages, ulong pos_dev, int batch, int steps, float scale);

    [LibraryImport(Library)]
    public static partial int ns_attention_decode_quant(nint dev, nint cache, ulong q, long q_stride, ulong o, long o_stride, ulong page_table, int max_pages, ulong pos_dev, int batch, int steps, float scale, ulong q_out, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_attention_prefill(nint dev, ulong q, ulong k, ulong v, ulong o, int batch, int heads, int seq, int head_dim, long* q_strides, long* k_strides, long* v_strides, long* o_strides, float scale, int causal);

    [LibraryImport(Library)]
    public static partial int ns_linear_create(nint dev, int K, int N, int mode, float* w_kn, float* bias, int split, int col_groups, int tp_rank, int tp_size, out nint linear);

    [LibraryImport(Library)]
    public static partial int ns_linear_create_bf16(nint dev, int N, int K, void* w_nk, out nint linear);

    [LibraryImport(Library)]
    public static partial int ns_linear_destroy(nint linear);

    [LibraryImport(Library)]
    public static partial int ns_linear_info(nint linear, int* k_local, int* n_local, int* mode, ulong* w, ulong* w_scale, ulong* bias);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward(nint dev, nint linear, ulong x, ulong x_scale, int M, int epilogue, ulong residual, int residual_dtype, int out_dtype, ulong y);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward_host(nint dev, nint linear, float* x_host, int M, int epilogue, float* y_host, int chunk_rows);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward_partial(nint dev, nint linear, ulong x, int M, out ulong partial, out int splits);

    [LibraryImport(Library)]
    public static partial int ns_finish_norm_quant(nint dev, ulong partial, int splits, nint linear, ulong x_scale, ulong residual, long rows, ulong x_out, ulong gamma, ulong beta, float eps, ulong q, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_finish_gelu_quant(nint dev, ulong partial, int splits, nint linear, ulong x_scale, long rows, ulong q, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_finish_kv_append(nint dev, ulong partial, int splits, nint linear, ulong x_scale, int batch, int steps, ulong qkv, nint cache, ulong page_table, int max_pages, ulong pos_dev);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward_norm_quant(nint dev, nint linear, ulong x, ulong x_scale, ulong residual, long rows, ulong x_out, ulong gamma, ulong beta, float eps, ulong q, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward_gelu_quant(nint dev, nint linear, ulong x, ulong x_scale, long rows, ulong q, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward_kv_append(nint dev, nint linear, ulong x, ulong x_scale, int batch, int steps, ulong qkv, nint cache, ulong page_table, int max_pages, ulong pos_dev);

    [LibraryImport(Library)]
    public static partial int ns_embed_ngram(nint dev, ulong ids, ulong table, int table_dtype, int table_ld, float scale, ulong bigram, int bigram_ld, int buckets, long mul_prev, long mul_cur, ulong slots, ulong last, int batch, int steps, int dim, int vocab, ulong y);

    [LibraryImport(Library)]
    public static partial int ns_rms_rows(nint dev, ulong x, ulong src, int splits, int src_dtype, int src_ld, float alpha, ulong x_out, ulong w, float eps, ulong row_map, long src_rows, long rows, int cols, int out_dtype, ulong y, int y_ld);

    [LibraryImport(Library)]
    public static partial int ns_rms_post_rows(nint dev, ulong x, ulong src, int splits, int src_dtype, int src_ld, ulong post_w, ulong plus, ulong x_out, ulong w, float eps, long rows, int cols, int out_dtype, ulong y, int y_ld);

    [LibraryImport(Library)]
    public static partial int ns_glu_rows(nint dev, ulong src, int splits, int src_dtype, int src_ld, long rows, int ff, int act, int out_dtype, ulong y, int y_ld);

    [LibraryImport(Library)]
    public static partial int ns_copy_cols(nint dev, ulong src, int splits, int src_dtype, int src_ld, int col, long rows, int cols, int out_dtype, ulong y, int y_ld);

    [LibraryImport(Library)]
    public static partial int ns_seq_advance(nint dev, ulong ids, ulong slots, int batch, int steps, ulong pos, ulong last);

    [LibraryImport(Library)]
    public static partial int ns_ids_from_f32(nint dev, ulong x, ulong ids, int n);

    [LibraryImport(Library)]
    public static partial int ns_short_conv(nint dev, ulong src, int splits, int src_dtype, int src_ld, int segments, long* fields, float* scales, long hist_slot_stride, ulong slots, ulong pos, int batch, int steps, int out_dtype);

    [LibraryImport(Library)]
    public static partial int ns_delta_recurrent(nint dev, ulong q, int q_ld, ulong k, int k_ld, ulong v, int v_ld, ulong a_src, int a_splits, int a_ld, int a_col, ulong b_src, int b_splits, int b_ld, int b_col, ulong a_log, ulong dt_bias, int per_channel, ulong state, long state_slot_stride, ulong slots, int batch, int steps, int heads, int kv_heads, int dim, int vdim, ulong o, int o_ld);

    [LibraryImport(Library)]
    public static partial int ns_delta_chunked(nint dev, ulong q, int q_ld, ulong k, int k_ld, ulong v, int v_ld, ulong a_src, int a_splits, int a_ld, int a_col, ulong b_src, int b_splits, int b_ld, int b_col, ulong a_log, ulong dt_bias, int per_channel, ulong state, long state_slot_stride, ulong slots, int batch, int steps, int heads, int kv_heads, int dim, int vdim, ulong o, int o_ld);

    [LibraryImport(Library)]
    public static partial int ns_gated_norm(nint dev, ulong o, int o_ld, ulong gate, int splits, int gate_dtype, int gate_ld, int gate_col, int act, ulong w, float eps, long rows, int heads, int vdim, int out_dtype, ulong y, int y_ld);

    [LibraryImport(Library)]
    public static partial int ns_lightning_recurrent(nint dev, ulong src, int splits, int src_dtype, int src_ld, int q_col, int k_col, int v_col, ulong decay, ulong decay_log2, ulong state, long state_slot_stride, ulong slots, int batch, int steps, int heads, int dim, int vdim, ulong o, int o_ld);

    [LibraryImport(Library)]
    public static partial int ns_lightning_chunked(nint dev, ulong src, int splits, int src_dtype, int src_ld, int q_col, int k_col, int v_col, ulong decay, ulong decay_log2, ulong state, long state_slot_stride, ulong slots, int batch, int steps, int heads, int dim, int vdim, ulong o, int o_ld, int segments);

    [LibraryImport(Library)]
    public static partial int ns_window_append(nint dev, ulong src, int splits, int src_dtype, int src_ld, int q_col, int k_col, int v_col, int g_col, int heads, int kv_heads, int dim, int vdim, ulong q_norm, ulong k_norm, float eps, ulong slots, ulong pos, int batch, int steps, int dtype, ulong q, ulong gate, ulong k_ring, ulong v_ring, long k_slot_stride, long v_slot_stride, int ring_len, int k_ld, int v_ld);

    [LibraryImport(Library)]
    public static partial int ns_window_attend(nint dev, int dtype, ulong q, ulong k_ring, ulong v_ring, long k_slot_stride, long v_slot_stride, int ring_len, int k_ld, int v_ld, ulong sink, ulong gate, ulong slots, ulong pos, int batch, int steps, int heads, int kv_heads, int dim, int vdim, int window, float scale, ulong o, long o_ld);

    [LibraryImport(Library)]
    public static partial int ns_window_decode(nint dev, ulong q, ulong k_ring, ulong v_ring, long k_slot_stride, long v_slot_stride, int ring_len, int k_ld, int v_ld, ulong sink, ulong gate, ulong slots, ulong pos, int batch, int steps, int heads, int kv_heads, int dim, int vdim, int window, float scale, ulong o, long o_ld);

    [LibraryImport(Library)]
    public static partial int ns_window_prefill(nint dev, ulong q, ulong k_ring, ulong v_ring, long k_slot_stride, long v_slot_stride, int slot_count, int ring_len, int k_ld, int v_ld, ulong sink, ulong gate, ulong slots, ulong pos, int batch, int steps, int heads, int kv_heads, int dim, int vdim, int window, float scale, ulong o, long o_ld);

    [LibraryImport(Library)]
    public static partial int ns_latent_append(nint dev, ulong src, int splits, int src_dtype, int src_ld, int q_rank, int kv_rank, int rot_dim, int rot_dims, ulong q_norm, ulong kv_norm, float eps, ulong freq, ulong slots, ulong pos, int batch, int steps, int dtype, ulong cq, int cq_ld, ulong ring, long ring_slot_stride, int ring_len, int ring_ld);

    [LibraryImport(Library)]
    public static partial int ns_rotate_heads(nint dev, ulong src, int splits, int src_dtype, int src_ld, int heads, int dim, int rot_dim, int rot_dims, ulong freq, ulong slots, ulong pos, int batch, int steps, int plain_dtype, ulong plain, long plain_ld, int plain_head, int rot_dtype, ulong rot, long rot_ld, int rot_head);

    [LibraryImport(Library)]
    public static partial int ns_head_matmul(nint dev, int x_dtype, ulong x, long x_ld, int x_head, int w_dtype, ulong w, long w_head, long w_k, long w_n, int y_dtype, ulong y, long y_ld, int y_head, int rows, int heads, int k, int n);

    [LibraryImport(Library)]
    public static partial int ns_latent_attend(nint dev, ulong q, int dtype, ulong ring, long ring_slot_stride, int ring_len, int ring_ld, int rank, int width, int window, float scale, ulong slots, ulong pos, int batch, int steps, int heads, ulong o);

    [LibraryImport(Library)]
    public static partial int ns_latent_decode(nint dev, ulong q, ulong ring, long ring_slot_stride, int ring_len, int ring_ld, int rank, int width, int window, float scale, ulong slots, ulong pos, int batch, int steps, int heads, ulong o);

    [LibraryImport(Library)]
    public static partial int ns_latent_gather(nint dev, ulong ring, long ring_slot_stride, int ring_len, int ring_ld, int past, ulong slots, ulong pos, int batch, int rows, ulong keys);

    [LibraryImport(Library)]
    public static partial int ns_latent_prefill(nint dev, ulong q, long q_ld, ulong kv, long kv_ld, ulong keys, long keys_ld, int rank, ulong slots, ulong pos, int batch, int steps, int heads, int dim, int rot_dim, int vdim, int past, int window, float scale, ulong o, long o_ld);

    [LibraryImport(Library)]
    public static partial int ns_bias_residual(nint dev, ulong partial, ulong bias, ulong residual, int residual_dtype, long rows, int cols, int out_dtype, ulong y);

    [LibraryImport(Library)]
    public static partial int ns_argmax_partial(nint dev, ulong x, int rows, int cols, long row_stride, int col_offset, ulong out_val, ulong out_idx);

    [LibraryImport(Library)]
    public static partial int ns_argmax_merge(nint dev, ulong vals, ulong idx, int parts, int rows, ulong ids);

    [LibraryImport(Library)]
    public static partial int ns_comm_unique_id(void* id128);

    [LibraryImport(Library)]
    public static partial int ns_comm_init_rank(nint dev, void* id128, int rank, int size, out nint comm);

    [LibraryImport(Library)]
    public static partial int ns_comm_info(nint comm, int* rank, int* size, int* nccl_version);

    [LibraryImport(Library)]
    public static partial int ns_allreduce(nint dev, nint comm, ulong buf, long count, int dtype);

    [LibraryImport(Library)]
    public static partial int ns_allgather(nint dev, nint comm, ulong src, ulong dst, long count, int dtype);

    [LibraryImport(Library)]
    public static partial int ns_comm_async_error(nint comm, out int nccl_result);

    [LibraryImport(Library)]
    public static partial int ns_comm_abort(nint comm);

    [LibraryImport(Library)]
    public static partial int ns_comm_destroy(nint comm);

    [LibraryImport(Library)]
    public static partial int ns_peer_group_create(nint dev, int rank, int world, ulong slot_bytes, out nint group);

    [LibraryImport(Library)]
    public static partial int ns_peer_group_handle(nint group, void* handle64);

    [LibraryImport(Library)]
    public static partial int ns_peer_group_connect(nint group, void* handles);

    [LibraryImport(Library)]
    public static partial int ns_peer_group_slot(nint group, int slot, out ulong ptr);

    [LibraryImport(Library)]
    public static partial int ns_tp_reduce_norm_quant(nint dev, nint group, int slot, ulong bias, ulong residual, long rows, int cols, ulong x_out, ulong gamma, ulong beta, float eps, ulong q, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_linear_forward_tp_norm_quant(nint dev, nint linear, nint group, int slot, ulong x, ulong x_scale, ulong residual, long rows, ulong x_out, ulong gamma, ulong beta, float eps, ulong q, ulong q_scale);

    [LibraryImport(Library)]
    public static partial int ns_peer_group_destroy(nint group);
}
