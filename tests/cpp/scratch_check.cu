// The library's host code against a CUDA runtime that only keeps books: every
// allocation, free and launch of an entry point, without a GPU.  Linked with
// the library's own objects in place of libcudart (tests/test_scratch.py).
// Allocations get addresses that are never used twice, a limit on their sum
// stands for the device's memory, and a stream (or another thread) can be
// declared to be capturing.
#include "kp_transport.cuh"

#include <cstdio>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace
{
struct launch_t
{
    std::string kernel;
    std::vector< void * > args;          // pointers among the arguments
    kp::fwd_params_t P;                  // ... of a kernel that takes one
};

struct
{
    std::map< uintptr_t, size_t > live;
    std::set< uintptr_t > freed;
    std::map< const void *, std::string > names;
    std::vector< launch_t > launches;
    uintptr_t next = 1ull << 40;
    size_t used = 0, limit = ~ ( size_t ) 0;
    cudaStream_t capturing = nullptr;    // the stream that is being captured
    bool other_captures = false;         // another thread captures, in the global mode
    bool broken = false;                 // a call that such a capture does not survive
    cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
    bool pending = false;                // no event is reached
    cudaError_t last = cudaSuccess;
    long calls = 0;

    bool unsafe(  )
    {
        const bool bad = mode != cudaStreamCaptureModeRelaxed && ( capturing || other_captures );
        broken = broken || bad;
        return bad;
    }
} F;

cudaError_t ret( cudaError_t e )
{
    ++ F.calls;
    if( e != cudaSuccess ) F.last = e;
    return e;
}

// The allocation that holds address a (0: none).
uintptr_t owner( uintptr_t a )
{
    auto it = F.live.upper_bound( a );
    if( it == F.live.begin(  ) ) return 0;
    -- it;
    return a < it->first + it->second ? it->first : 0;
}

int fails = 0;
void expect( bool ok, const char * what )
{
    if( ! ok ) { std::printf( "FAIL %s\n", what ); ++ fails; }
}
}   // namespace

void register_linked( void ( * cb )( void ** ), void *, void *, void ( * )( void * ) )
{
    static void * handle[ 2 ];
    cb( handle );
}

#ifndef __CUDA_ARCH__                  // the device pass declares the runtime for kernels
extern "C" {
void fake_register( void ( * cb )( void ** ), void * a, void * b, void ( * c )( void * ) ) { register_linked( cb, a, b, c ); }
void __cudaRegisterFunction( void **, const char * host, char *, const char * name, int, uint3 *, uint3 *, dim3 *, dim3 *, int * )
{ F.names[ host ] = name; }
void ** __cudaRegisterFatBinary( void * ) { static void * handle[ 2 ]; return handle; }
void __cudaRegisterFatBinaryEnd( void ** ) {  }
void __cudaUnregisterFatBinary( void ** ) {  }
void __cudaRegisterVar( void **, char *, char *, const char *, int, size_t, int, int ) {  }
static struct { dim3 g, b; size_t sh; cudaStream_t s; } conf;
unsigned __cudaPushCallConfiguration( dim3 g, dim3 b, size_t sh, cudaStream_t s ) { conf = { g, b, sh, s }; return 0; }
cudaError_t __cudaPopCallConfiguration( dim3 * g, dim3 * b, size_t * sh, void * s )
{ * g = conf.g; * b = conf.b; * sh = conf.sh; * ( cudaStream_t * ) s = conf.s; return cudaSuccess; }
cudaError_t cudaLaunchKernel( const void * f, dim3, dim3, void ** args, size_t, cudaStream_t )
{
    launch_t l {  };
    l.kernel = F.names[ f ];
    if( l.kernel.find( "12fwd_params_t" ) != std::string::npos )
    {
        std::memcpy( & l.P, args[ 0 ], sizeof( l.P ) );
        if( l.kernel.find( "k_task_sort" ) != std::string::npos )
            for( int k = 1; k < 3; ++ k ) l.args.push_back( * ( void ** ) args[ k ] );
    }
    F.launches.push_back( l );
    return ret( cudaSuccess );
}
cudaError_t cudaMalloc( void ** p, size_t n )
{
    * p = nullptr;
    if( F.unsafe(  ) ) return ret( cudaErrorStreamCaptureUnsupported );
    if( F.used + n > F.limit ) return ret( cudaErrorMemoryAllocation );
    * p = ( void * ) F.next;
    F.live[ F.next ] = n;
    F.used += n;
    F.next += ( n + 4095 ) / 4096 * 4096 + 4096;
    return ret( cudaSuccess );
}
cudaError_t cudaFree( void * p )
{
    if( p == nullptr ) return ret( cudaSuccess );
    if( F.unsafe(  ) ) return ret( cudaErrorStreamCaptureUnsupported );
    auto it = F.live.find( ( uintptr_t ) p );
    expect( it != F.live.end(  ), "a free of what is not allocated" );
    if( it == F.live.end(  ) ) return ret( cudaErrorInvalidValue );
    F.used -= it->second;
    F.freed.insert( it->first );
    F.live.erase( it );
    return ret( cudaSuccess );
}
cudaError_t cudaStreamIsCapturing( cudaStream_t s, cudaStreamCaptureStatus * st )
{
    * st = F.capturing && s == F.capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return ret( cudaSuccess );
}
cudaError_t cudaThreadExchangeStreamCaptureMode( cudaStreamCaptureMode * m ) { std::swap( * m, F.mode ); return ret( cudaSuccess ); }
cudaError_t cudaGetLastError( void ) { const auto e = F.last; F.last = cudaSuccess; ++ F.calls; return e; }
cudaError_t cudaPeekAtLastError( void ) { return F.last; }
const char * cudaGetErrorString( cudaError_t e ) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDevice( int * d ) { * d = 0; return ret( cudaSuccess ); }
cudaError_t cudaSetDevice( int ) { return ret( cudaSuccess ); }
cudaError_t cudaGetDeviceCount( int * n ) { * n = 1; return ret( cudaSuccess ); }
cudaError_t cudaDeviceGetAttribute( int * v, cudaDeviceAttr, int ) { * v = 148; return ret( cudaSuccess ); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor( int * n, const void *, int, size_t ) { * n = 5; return ret( cudaSuccess ); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags( int * n, const void *, int, size_t, unsigned ) { * n = 5; return ret( cudaSuccess ); }
cudaError_t cudaFuncGetAttributes( cudaFuncAttributes * a, const void * )
{ * a = cudaFuncAttributes {  }; a->ptxVersion = a->binaryVersion = 100; return ret( cudaSuccess ); }
cudaError_t cudaMemset( void *, int, size_t ) { return ret( cudaSuccess ); }
cudaError_t cudaMemsetAsync( void *, int, size_t, cudaStream_t ) { return ret( cudaSuccess ); }
cudaError_t cudaMemcpy( void *, const void *, size_t, cudaMemcpyKind ) { return ret( cudaSuccess ); }
cudaError_t cudaMemcpyAsync( void *, const void *, size_t, cudaMemcpyKind, cudaStream_t ) { return ret( cudaSuccess ); }
cudaError_t cudaEventCreateWithFlags( cudaEvent_t * e, unsigned ) { * e = nullptr; return ret( cudaSuccess ); }
cudaError_t cudaEventDestroy( cudaEvent_t ) { return ret( cudaSuccess ); }
cudaError_t cudaEventRecord( cudaEvent_t, cudaStream_t ) { return ret( cudaSuccess ); }
cudaError_t cudaEventQuery( cudaEvent_t ) { return F.unsafe(  ) ? ret( cudaErrorStreamCaptureUnsupported ) : ret( F.pending ? cudaErrorNotReady : cudaSuccess ); }
cudaError_t cudaStreamGetId( cudaStream_t s, unsigned long long * id ) { * id = ( unsigned long long ) s; return ret( cudaSuccess ); }
cudaError_t cudaStreamWaitEvent( cudaStream_t, cudaEvent_t, unsigned ) { return ret( cudaSuccess ); }
cudaError_t cudaDeviceSynchronize( void ) { return ret( cudaSuccess ); }
cudaError_t cudaStreamSynchronize( cudaStream_t ) { return ret( cudaSuccess ); }
}   // extern "C"
#endif

namespace
{
struct solve_t
{
    kp_transport_cfg_t cfg {  };
    kp_tallies_t t {  };
    kp_source_t src { KP_SOURCE_POINT, KP_EMIT_ISOTROPIC, { 0.5, 0.5, 0.5 } };
    solve_t( long long n, bool image )
    {
        cfg.n_packets = n;
        cfg.n_sources = 1;
        cfg.sources = & src;
        cfg.max_scatter = 100;
        cfg.max_steps = 100000;
        cfg.fx_shift = 32;
        cfg.n_batches = cfg.image_batch_n = 1;
        cfg.image_n = image ? 32 : 0;
        cfg.image_half_width = 1;
        cfg.inclination_deg = 60;
        cfg.image_center[ 0 ] = cfg.image_center[ 1 ] = cfg.image_center[ 2 ] = 0.5;
        t.image = t.image_batch = ( void * ) 4096;
    }
    // a float flux with its carry, on a mesh of n cells
    solve_t & flux( long long n )
    {
        cfg.tally_mode = KP_TALLY_FLOAT;
        t.flux = t.carry = ( float * ) 4096;
        t.flux_n = n;
        return * this;
    }
    int run( kp_mesh_t * m, cudaStream_t s = nullptr ) { return kp_transport_forward( m, & cfg, & t, s ); }
    long long tape( kp_mesh_t * m )
    {
        long long id = 0;
        expect( kp_transport_forward_tape( m, & cfg, & t, nullptr, & id ) == KP_OK && id > 0, "taped solve" );
        return id;
    }
    int adjoint( kp_mesh_t * m, cudaStream_t s )
    { return kp_transport_adjoint( m, & cfg, ( float * ) 4096, 24, ( void * ) 4096, ( void * ) 4096, nullptr, s ); }
    int adjoint_tape( kp_mesh_t * m, long long id )
    { return kp_transport_adjoint_tape( m, id, & cfg, ( float * ) 4096, 24, ( void * ) 4096, ( void * ) 4096, nullptr, nullptr ); }
};

// A uniform mesh of n^3 cells in blocks of 16^3.
kp_mesh_t * make_mesh( int n )
{
    kp_mesh_desc_t d {  };
    for( int a = 0; a < 3; ++ a )
    {
        d.x_max[ a ] = 1;
        d.n_cell_global[ a ] = n;
        d.n_cell_block[ a ] = 16;
    }
    kp_mesh_t * m = nullptr;
    expect( kp_mesh_create( & d, & m ) == KP_OK, "mesh" );
    return m;
}

// A mesh that was never on a device comes and goes without the runtime, whose
// first call (a free of null is one) would make a context.
void host_mesh(  )
{
    kp_mesh_destroy( make_mesh( 32 ) );
    expect( F.calls == 0, "a host mesh calls the runtime" );
}

// The gradient of a taped solve has room for its walk's packets, or an error.
void tape_pool(  )
{
    kp_mesh_t * m = make_mesh( 32 );
    solve_t taped( 2000, true ), plain( 100000, false );
    const long long id = taped.tape( m );
    F.limit = 0;                         // the device is full, another program's what is freed
    plain.run( m );
    F.launches.clear(  );
    const int r = taped.adjoint_tape( m, id );
    bool walked = false;
    for( const auto & l : F.launches )
        if( l.kernel.find( "k_walk" ) != std::string::npos )
            walked = l.P.pool != nullptr && l.P.pool_n > 0;
    expect( r != KP_OK || walked, "adjoint without a pool" );
    kp_mesh_destroy( m );
}
// The allocations that the launches so far were given.
std::set< uintptr_t > given(  )
{
    std::set< uintptr_t > r;
    for( const auto & l : F.launches )
    {
        std::vector< uintptr_t > w( sizeof( l.P ) / sizeof( uintptr_t ) );
        std::memcpy( w.data(  ), & l.P, w.size(  ) * sizeof( uintptr_t ) );
        for( void * a : l.args ) w.push_back( ( uintptr_t ) a );
        for( uintptr_t a : w ) if( owner( a ) ) r.insert( owner( a ) );
    }
    return r;
}

// What a captured solve was given stays allocated, through larger solves and a
// lower queue limit, until its mesh goes; the larger solves' own buffers are
// not kept beside it.
void captured(  )
{
    const cudaStream_t S = ( cudaStream_t ) 64;
    for( int kind = 0; kind < 4; ++ kind )           // as queued, by cell, adjoint, no image
    {
        kp_mesh_t * m = make_mesh( 32 );
        if( kind == 1 ) kp_mesh_peel_order( m, KP_PEEL_ORDER_CELL );
        auto solve = [ & ]( long long n )
        {
            solve_t s( n, kind != 3 );
            return kind == 2 ? s.adjoint( m, S ) : s.run( m, S );
        };
        solve_t image( 20000, true );                // a queue and adjoint buffers beside it
        expect( image.run( m, S ) == KP_OK && image.adjoint( m, S ) == KP_OK, "solve" );
        expect( solve( 20000 ) == KP_OK, "solve" );
        F.capturing = S;
        F.launches.clear(  );
        expect( solve( 20000 ) == KP_OK && ! F.broken, "captured solve" );
        F.capturing = nullptr;
        const auto held = given(  );
        size_t n_live = 0;
        for( int k = 0; k < 3; ++ k )
        {
            expect( solve( 100000 << k ) == KP_OK, "larger solve" );
            if( k > 0 ) expect( F.live.size(  ) <= n_live, "outgrown buffers pile up" );
            n_live = F.live.size(  );
        }
        solve_t larger( 500000, true );
        expect( larger.adjoint( m, S ) == KP_OK, "larger solve" );
        expect( m->kept.size(  ) == ( kind == 0 ? 1 : kind == 3 ? 0 : 2 ), "kept: what the capture was given, no more" );
        expect( kp_mesh_peel_queue_limit( m, 5000 ) == KP_OK && solve( 1000 ) == KP_OK, "lower limit" );
        for( uintptr_t a : held )
            expect( F.live.count( a ) != 0, "a captured solve's memory was freed" );
        kp_mesh_destroy( m );
        expect( F.live.size(  ) <= 1, "memory left behind" );     // a pool to be lent
    }
}
// Where the packet count chooses the march order, it does so at the stated count
// and only where the caller left the choice.
void order_by_count(  )
{
    kp_mesh_t * m = make_mesh( 160 );                // 16 MB of extinction
    auto sorted = [ & ]( int order, long long n )
    {
        kp_mesh_peel_order( m, order );
        F.launches.clear(  );
        expect( solve_t( n, true ).run( m ) == KP_OK, "solve" );
        int sorts = 0, marches = 0;
        for( const auto & l : F.launches )
        {
            sorts += l.kernel.find( "k_task_sort" ) != std::string::npos;
            marches += l.kernel.find( "k_peel" ) != std::string::npos && l.P.pq_perm != nullptr;
        }
        expect( sorts == 2 * marches, "sorted and marched so" );
        return marches == 1;
    };
    expect( ! sorted( KP_PEEL_ORDER_AUTO, KP_PEEL_SORT_MANY - 1 ), "as queued below the count" );
    expect( sorted( KP_PEEL_ORDER_AUTO, KP_PEEL_SORT_MANY ), "by cell from the count on" );
    expect( ! sorted( KP_PEEL_ORDER_AUTO, 1000 ), "as queued again" );
    expect( ! sorted( KP_PEEL_ORDER_QUEUE, KP_PEEL_SORT_MANY ) && sorted( KP_PEEL_ORDER_CELL, 1000 ), "the caller's order" );
    kp_mesh_destroy( m );
}

// What a solve allocates beside its queue, for speed alone, disturbs no capture
// under way in another thread, and a captured solve has it too.
void other_capture(  )
{
    kp_mesh_t * m = make_mesh( 160 );                // 16 MB of extinction: sorted by the packet count
    solve_t s( 500000, true );
    kp_mesh_peel_order( m, KP_PEEL_ORDER_QUEUE );
    expect( s.run( m ) == KP_OK, "solve as queued" );
    kp_mesh_peel_order( m, KP_PEEL_ORDER_AUTO );
    F.other_captures = true;
    F.launches.clear(  );
    expect( s.run( m ) == KP_OK && ! F.broken, "the march order's buffers" );
    bool sorted = false;
    for( const auto & l : F.launches ) sorted = sorted || l.kernel.find( "k_task_sort" ) != std::string::npos;
    expect( sorted, "marched by cell" );
    F.other_captures = false;
    kp_mesh_destroy( m );

    for( const cudaStream_t S : { ( cudaStream_t ) nullptr, ( cudaStream_t ) 64 } )
    {
        m = make_mesh( 32 );
        solve_t f( 2000, false );
        expect( f.run( m ) == KP_OK, "solve" );
        F.capturing = S;                             // itself captured, or beside a capture
        F.other_captures = S == nullptr;
        F.launches.clear(  );
        f.flux( 32768 );
        expect( f.run( m, S ) == KP_OK && ! F.broken, "the flux sums" );
        for( const auto & l : F.launches )
            expect( l.kernel.find( "k_walk" ) == std::string::npos || l.P.flux_sum, "flux in double" );
        F.capturing = nullptr;
        F.other_captures = false;
        kp_mesh_destroy( m );
    }
}
// The packet pools of the launches so far.
std::set< uintptr_t > pools(  )
{
    std::set< uintptr_t > r;
    for( const auto & l : F.launches )
        if( owner( ( uintptr_t ) l.P.pool ) ) r.insert( owner( ( uintptr_t ) l.P.pool ) );
    return r;
}

// A mesh's first solve without an image allocates nothing where another's pool
// is free; solves in flight on several streams have pools of their own.
void first_solve(  )
{
    const cudaStream_t A = ( cudaStream_t ) 64, B = ( cudaStream_t ) 128;
    std::vector< kp_mesh_t * > m;
    auto solve = [ & ]( cudaStream_t s, long long n )
    {
        m.push_back( make_mesh( 32 ) );
        expect( kp_mesh_upload( m.back(  ) ) == KP_OK, "upload" );
        const size_t before = F.used;
        F.launches.clear(  );
        expect( solve_t( n, false ).run( m.back(  ), s ) == KP_OK && pools(  ).size(  ) == 1, "solve" );
        return F.used - before;
    };
    expect( solve( A, 2000 ) > 0, "the first of all" );
    const auto one = pools(  );
    F.pending = true;                                // no solve ends
    for( int k = 0; k < 8; ++ k ) expect( solve( A, 100000 << k % 3 ) == 0 && pools(  ) == one, "a pool in stream order" );
    expect( solve( B, 2000 ) > 0 && pools(  ) != one, "two streams, two pools" );
    expect( solve( A, 2000 ) == 0 && solve( B, 2000 ) == 0, "two pools for two streams" );
    F.pending = false;
    expect( solve( ( cudaStream_t ) 192, 2000000 ) == 0, "a third stream once they have ended" );
    for( auto * p : m ) kp_mesh_destroy( p );
    expect( F.live.size(  ) == 1, "one pool is left" );
}

// A solve that fits the device without what is kept for speed alone (packet
// pools, flux sums, the order by packet count) runs, whatever came before it.
void short_memory(  )
{
    constexpr size_t SLACK = 1 << 16;                // a block's packets
    for( int kind = 0; kind < 4; ++ kind )           // as queued, by cell, adjoint, tape
    {
        auto order = [ & ]( kp_mesh_t * m ) { if( kind == 1 ) kp_mesh_peel_order( m, KP_PEEL_ORDER_CELL ); };
        auto solve = [ & ]( kp_mesh_t * m )
        {
            solve_t s( 100000, true );
            if( kind < 2 ) s.flux( 64 * 64 * 64 );
            return kind == 2 ? s.adjoint( m, nullptr ) : kind == 3 ? ( s.tape( m ), ( int ) KP_OK ) : s.run( m );
        };
        kp_mesh_t * m = make_mesh( 64 );
        order( m );
        expect( solve( m ) == KP_OK, "solve" );
        size_t need = F.used - ( m->d_flux ? 64 * 64 * 64 * 8 : 0 );
        for( uintptr_t a : pools(  ) ) need -= F.live[ a ];
        kp_mesh_destroy( m );
        for( int before = 0; before < 2; ++ before )
        {
            m = make_mesh( 64 );
            order( m );
            if( before )
            {   // a pool, flux sums and a small queue of earlier solves
                solve_t a( 50000, false ), b( 100, true );
                expect( a.flux( 64 * 64 * 64 ).run( m ) == KP_OK && b.run( m ) == KP_OK, "earlier solves" );
            }
            F.limit = need + SLACK;
            F.launches.clear(  );
            expect( solve( m ) == KP_OK, "a solve that fits" );
            for( const auto & l : F.launches )
                if( l.kernel.find( "k_walk" ) != std::string::npos )
                    expect( owner( ( uintptr_t ) l.P.pool ) && ( ! l.P.flux_sum || owner( ( uintptr_t ) l.P.flux_sum ) ),
                            "the walk's memory" );
            F.limit = ~ ( size_t ) 0;
            F.last = cudaSuccess;
            kp_mesh_destroy( m );
            expect( F.live.size(  ) <= 1, "memory left behind" );
        }
    }
    // an order by the packet count that a capture was given, and no memory for
    // a larger solve's: that one marches as queued, the capture keeps its own
    const cudaStream_t S = ( cudaStream_t ) 64;
    kp_mesh_t * m = make_mesh( 160 );
    solve_t s( 500000, true ), larger( 600000, true );
    expect( s.run( m, S ) == KP_OK, "solve" );
    F.capturing = S;
    F.launches.clear(  );
    expect( s.run( m, S ) == KP_OK && ! F.broken, "captured solve" );
    F.capturing = nullptr;
    const auto held = given(  );
    F.limit = F.used + 600000ull * 12 * 64 + SLACK;
    expect( larger.run( m, S ) == KP_OK, "larger solve" );
    for( uintptr_t a : held )
        expect( F.live.count( a ) != 0, "a captured order was freed" );
    kp_mesh_destroy( m );
}
// A trace's shares hold every packet once, and packets that lie together in
// the pool are many warps'.
void shares(  )
{
    for( const long long w : { 4ll, 2960ll, 3552ll } )
        for( const long long n : { 1ll, 31ll, 2001ll, 47359ll, 47360ll, 100003ll, 300001ll, 1048576ll } )
        {
            const kp::share_t s = kp::share_t::make( n, w, 4 );
            std::vector< char > seen( n );
            long long longest = 0, front = 0;        // of a share, and of its packets in the first eighth
            for( long long k = 0; k < w; ++ k )
            {
                long long of_front = 0;
                for( long long at = 0; at < s.size( k ); ++ at )
                    if( const long long i = s.item( k, at ); i < n )
                    {
                        expect( ! seen[ i ], "a packet of two shares" );
                        seen[ i ] = 1;
                        of_front += i < n / 8;
                    }
                longest = std::max( longest, s.size( k ) );
                front = std::max( front, of_front );
            }
            for( char c : seen ) if( ! c ) { expect( false, "a packet of no share" ); break; }
            expect( longest <= n / w + n / w / 16 + 2, "an even share" );
            expect( front <= n / 8 / w + ( 1 << s.unit ), "the pool's front in few shares" );
        }
}
}   // namespace

int main( int argc, char ** argv )
{
    const std::string what = argc > 1 ? argv[ 1 ] : "";
    if( what == "host_mesh" ) host_mesh(  );
    else if( what == "tape_pool" ) tape_pool(  );
    else if( what == "captured" ) captured(  );
    else if( what == "other_capture" ) other_capture(  );
    else if( what == "short_memory" ) short_memory(  );
    else if( what == "shares" ) shares(  );
    else if( what == "order_by_count" ) order_by_count(  );
    else if( what == "first_solve" ) first_solve(  );
    else return 2;
    if( fails == 0 ) std::printf( "OK %s\n", what.c_str(  ) );
    return fails != 0;
}
