// Geometric walk with the path-length flux estimator, reference semantics.
//
// A packet walks cell by cell until its step budget runs out or it leaves
// the domain, exactly as photon::cart_t::proc does
// (modules/particle/radiation/photon.h:104-125) when integrate::ker_itg runs
// it over the pool (evolve/integrator.h:80-106).  Every floating-point
// operation rounds as the reference's does in its order, so that results
// equal the reference compiled for the host with contraction off, bit for
// bit, in FP32 (PRECISION=1) and FP64 (PRECISION=2).  Packet state is
// structure-of-arrays instead of the reference's 56-byte AoS pool records.
#include "kp_common.cuh"

#include <cfloat>

namespace kp
{
namespace
{

constexpr int8_t TO_KEEP = -2;      // particle::todo_t, types/particle_base.h:12
constexpr int8_t TO_RM   = -3;

// Round-to-nearest arithmetic without contraction, per float type.
__device__ __forceinline__ float  rn_add( float a, float b )   { return __fadd_rn( a, b ); }
__device__ __forceinline__ float  rn_sub( float a, float b )   { return __fsub_rn( a, b ); }
__device__ __forceinline__ float  rn_mul( float a, float b )   { return __fmul_rn( a, b ); }
__device__ __forceinline__ float  rn_div( float a, float b )   { return __fdiv_rn( a, b ); }
__device__ __forceinline__ double rn_add( double a, double b ) { return __dadd_rn( a, b ); }
__device__ __forceinline__ double rn_sub( double a, double b ) { return __dsub_rn( a, b ); }
__device__ __forceinline__ double rn_mul( double a, double b ) { return __dmul_rn( a, b ); }
__device__ __forceinline__ double rn_div( double a, double b ) { return __ddiv_rn( a, b ); }

template< class f_t > struct geo_ptr;
template<> struct geo_ptr< float >
{ static __device__ const float * get( const mesh_view_t & m ) { return m.geo_f; } };
template<> struct geo_ptr< double >
{ static __device__ const double * get( const mesh_view_t & m ) { return m.geo_d; } };

template< class f_t > __device__ __forceinline__ int geo_stride(  );
template<> __device__ __forceinline__ int geo_stride< float  >(  ) { return 8; }
template<> __device__ __forceinline__ int geo_stride< double >(  ) { return 16; }
template< class f_t > __device__ __forceinline__ f_t xlim( const mesh_view_t & m, int l, int a );
template<> __device__ __forceinline__ float  xlim< float  >( const mesh_view_t & m, int l, int a ) { return m.xlim_f[ l ][ a ]; }
template<> __device__ __forceinline__ double xlim< double >( const mesh_view_t & m, int l, int a ) { return m.xlim_d[ l ][ a ]; }
template< class f_t > __device__ __forceinline__ f_t lbox( const mesh_view_t & m, int a );
template<> __device__ __forceinline__ float  lbox< float  >( const mesh_view_t & m, int a ) { return m.lbox_f[ a ]; }
template<> __device__ __forceinline__ double lbox< double >( const mesh_view_t & m, int a ) { return m.lbox_d[ a ]; }

// Block geometry (geo_t with uniform spacing, geometry.h:199-256).
template< class f_t >
struct blk_geo_t
{
    f_t xf0[ 3 ], dx0[ 3 ], vol0;
    __device__ void load( const mesh_view_t & m, int b )
    {
        const f_t * g = geo_ptr< f_t >::get( m ) + geo_stride< f_t >(  ) * ( size_t ) b;
        #pragma unroll
        for( int a = 0; a < 3; ++ a ) { xf0[ a ] = g[ a ]; dx0[ a ] = g[ 3 + a ]; }
        vol0 = g[ 6 ];
    }
    // geo_t::x_fc for uniform blocks (geometry.h:206-221)
    __device__ __forceinline__ f_t x_fc( int a, int i ) const
    {
        return rn_add( xf0[ a ], rn_mul( ( f_t ) i, dx0[ a ] ) );
    }
};

// particle::geo_loc_t (types/particle_base.h:86-126), including fix()'s
// use of the unchanged cell index when it re-snaps.
template< class f_t >
struct geo_loc_t
{
    f_t x_l[ 3 ], x_r[ 3 ];
    __device__ __forceinline__ void load( const blk_geo_t< f_t > & g, const int i[ 3 ] )
    {
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
        {
            x_l[ a ] = g.x_fc( a, i[ a ] );
            x_r[ a ] = g.x_fc( a, i[ a ] + 1 );
        }
    }
    __device__ __forceinline__ void shift( const blk_geo_t< f_t > & g, const int i[ 3 ],
                                           int ax, bool rhs )
    {
        #pragma unroll
        for( int a = 0; a < 3; ++ a )   // static indexing keeps x_l/x_r in registers
            if( a == ax )
            {
                if( rhs ) { x_l[ a ] = x_r[ a ]; x_r[ a ] = g.x_fc( a, i[ a ] + 1 ); }
                else      { x_r[ a ] = x_l[ a ]; x_l[ a ] = g.x_fc( a, i[ a ] ); }
            }
    }
    __device__ __forceinline__ void fix( const blk_geo_t< f_t > & g, const int i[ 3 ],
                                         const f_t x[ 3 ] )
    {
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
            if( x[ a ] > x_r[ a ] )      shift( g, i, a, true );
            else if( x[ a ] < x_l[ a ] ) shift( g, i, a, false );
    }
};

// One packet walked to its end, step by step as photon::cart_t::proc does
// (modules/particle/radiation/photon.h:104-125).  k_trace's walk is this one
// with its invariants kept in registers; the packets it cannot take (a
// starting cell outside its block, a direction whose reciprocal could leave
// the normal range) come here.
template< class f_t, int FLUX >
__device__ __noinline__ void trace_one( const mesh_view_t & m, long long p, f_t * __restrict__ xs,
                                        const f_t * __restrict__ dirs, int * __restrict__ cells,
                                        int * __restrict__ ibs, const f_t * __restrict__ propers,
                                        int * __restrict__ steps, int8_t * __restrict__ todos,
                                        void * __restrict__ flux, double fx_scale )
{
    f_t x[ 3 ], dir[ 3 ];
    int i[ 3 ];
    #pragma unroll
    for( int a = 0; a < 3; ++ a )
    {
        x  [ a ] = xs  [ 3 * p + a ];
        dir[ a ] = dirs[ 3 * p + a ];
        i  [ a ] = cells[ 3 * p + a ];
    }
    int ib   = ibs  [ p ];
    int step = steps[ p ];
    const f_t proper = propers[ p ];
    int8_t todo = -1;                       // dest.i_rank = -1 (photon.h:108)

    if( ib < 0 || ib >= m.n_blocks )
    {
        atomicOr( m.status, ST_BAD_BLOCK );
        return;
    }

    blk_geo_t< f_t > g;
    geo_loc_t< f_t > gl;
    int ib_old = -1;
    for( ; step > 0; -- step )
    {
        if( ib != ib_old && ib >= 0 )
        {   // photon.h:113-118
            g.load( m, ib );
            gl.load( g, i );
            gl.fix( g, i, x );
            ib_old = ib;
        }
        // proc_step (photon.h:85-102) with prx = bmap[ib] bound here.
        const int ib_cur = ib;
        // get_dl (photon.h:20-44)
        f_t dl[ 3 ];
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
        {
            if( dir[ a ] == 0 ) { dl[ a ] = -1; continue; }
            const f_t x_f = dir[ a ] > 0 ? gl.x_r[ a ] : gl.x_l[ a ];
            dl[ a ] = rn_div( rn_sub( x_f, x[ a ] ), dir[ a ] );
        }
        int a_proc = 0;
        f_t dl_min = ( f_t ) FLT_MAX;
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
            if( dl[ a ] >= 0 && dl[ a ] <= dl_min ) { a_proc = a; dl_min = dl[ a ]; }
        f_t dl_p = dl[ 0 ];
        #pragma unroll
        for( int a = 1; a < 3; ++ a ) if( a == a_proc ) dl_p = dl[ a ];

        // proc_phys (photon.h:73-83): flux += proper * dl / volume
        {
            const f_t dsi = rn_div( dl_p, g.vol0 );
            const f_t v   = rn_mul( proper, dsi );
            const bool in = i[ 0 ] >= 0 && i[ 0 ] < m.nc[ 0 ] &&
                            i[ 1 ] >= 0 && i[ 1 ] < m.nc[ 1 ] &&
                            i[ 2 ] >= 0 && i[ 2 ] < m.nc[ 2 ];
            if( ! in )
                atomicOr( m.status, ST_BAD_CELL );
            else
            {
                const size_t c = ( size_t ) ib_cur * m.cpb + i[ 0 ] +
                                 m.nc[ 0 ] * ( i[ 1 ] + m.nc[ 1 ] * i[ 2 ] );
                if( FLUX == KP_FLUX_FLOAT )
                    atomicAdd( ( f_t * ) flux + c, v );
                else
                    atomicAdd( ( unsigned long long * ) flux + c,
                               ( unsigned long long ) __double2ll_rn(
                                   ( double ) v * fx_scale ) );
            }
        }
        // proc_geo (photon.h:54-71)
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
        {
            if( a == a_proc )
            {
                const bool rhs = dir[ a ] > 0;
                x[ a ] = rhs ? gl.x_r[ a ] : gl.x_l[ a ];
                i[ a ] += rhs ? 1 : -1;
                gl.shift( g, i, a, rhs );
            }
            else
                x[ a ] = rn_add( x[ a ], rn_mul( dl_p, dir[ a ] ) );
        }
        // proxy_base_t::shift_blk (types/proxy.h:64-121) on block ib_cur
        todo = TO_KEEP;
        {
            const blk_meta_t md = m.meta[ ib_cur ];
            #pragma unroll
            for( int a = 0; a < 3; ++ a )
            {
                if( i[ a ] >= 0 && i[ a ] < m.nc[ a ] )
                    continue;
                const int side = i[ a ] > 0;
                if( ( md.phybnd >> ( 2 * a + side ) ) & 1 )
                {
                    todo = TO_RM;
                    break;
                }
                const int ap0 = a == 2 ? 0 : a + 1;
                const int ap1 = a == 0 ? 2 : a - 1;   // (a + 2) % 3
                const int dlv = md.d_lvl[ 2 * a + side ];
                int j0 = 0, j1 = 0;
                if( dlv > 0 )
                {
                    j0 = i[ ap0 ] >= m.nc[ ap0 ] / 2;
                    j1 = i[ ap1 ] >= m.nc[ ap1 ] / 2;
                }
                const int nid = m.nb[ 24 * ( size_t ) ib_cur +
                                      ( ( a * 2 + side ) * 2 + j0 ) * 2 + j1 ];
                ib = nid;
                if( nid < 0 )
                {
                    todo = TO_RM;
                    break;
                }
                i[ a ] = i[ a ] > 0 ? 0 : m.nc[ a ] - 1;
                const int sh = md.shift[ 2 * a + side ];
                if( dlv < 0 )
                {
                    i[ ap0 ] = i[ ap0 ] / 2 + ( sh & 1 ) * m.nc[ ap0 ] / 2;
                    i[ ap1 ] = i[ ap1 ] / 2 + ( ( sh >> 1 ) & 1 ) * m.nc[ ap1 ] / 2;
                }
                else if( dlv > 0 )
                {
                    const int h0 = m.nc[ ap0 ] / 2, h1 = m.nc[ ap1 ] / 2;
                    i[ ap0 ] = ( i[ ap0 ] < h0 ? i[ ap0 ] : i[ ap0 ] - h0 ) * 2;
                    i[ ap1 ] = ( i[ ap1 ] < h1 ? i[ ap1 ] : i[ ap1 ] - h1 ) * 2;
                }
                break;
            }
        }
        const bool proc_flag = todo != TO_RM;
        // par_base_t::regulate (particle_base.h:37-56), always evaluated
        bool wrapped = false;
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
            if( ( m.periodic >> a ) & 1 )
            {
                if( x[ a ] < xlim< f_t >( m, 0, a ) )
                {
                    x[ a ] = rn_add( x[ a ], lbox< f_t >( m, a ) );
                    wrapped = true;
                }
                else if( x[ a ] >= xlim< f_t >( m, 1, a ) )
                {
                    x[ a ] = rn_sub( x[ a ], lbox< f_t >( m, a ) );
                    wrapped = true;
                }
            }
        if( proc_flag && wrapped )
        {
            if( ib < 0 || ib >= m.n_blocks )
            {
                atomicOr( m.status, ST_BAD_BLOCK );
                todo = TO_RM;
                break;
            }
            g.load( m, ib );
            gl.load( g, i );
            gl.fix( g, i, x );
            ib_old = ib;   // geo_loc now describes block ib
        }
        if( ! proc_flag )
            break;
        if( ib < 0 || ib >= m.n_blocks )
        {
            atomicOr( m.status, ST_BAD_BLOCK );
            todo = TO_RM;
            break;
        }
    }
    if( step <= 0 )
        todo = TO_RM;

    #pragma unroll
    for( int a = 0; a < 3; ++ a )
    {
        xs   [ 3 * p + a ] = x[ a ];
        cells[ 3 * p + a ] = i[ a ];
    }
    ibs  [ p ] = ib;
    steps[ p ] = step;
    todos[ p ] = todo;
}

// a / b for a divisor whose correctly rounded reciprocal y is at hand: two
// remainder corrections of a y give the correctly rounded quotient (Markstein,
// IBM J. Res. Dev. 34, 1990), the value of rn_div, in five multiply-adds.
// Holds while nothing leaves the normal range; quot_range bounds |a| from below
// (the remainder is then normal), the callers bound b, and a quotient that
// overflows comes out as NaN.
template< class f_t > struct quot_range;
template<> struct quot_range< float >
{ static __device__ __forceinline__ float  lo(  ) { return 0x1p-62f; } static __device__ __forceinline__ float  hi(  ) { return 0x1p62f; } };
template<> struct quot_range< double >
{ static __device__ __forceinline__ double lo(  ) { return 0x1p-480; } static __device__ __forceinline__ double hi(  ) { return 0x1p480; } };
__device__ __forceinline__ float  rn_fma( float a, float b, float c )    { return __fmaf_rn( a, b, c ); }
__device__ __forceinline__ double rn_fma( double a, double b, double c ) { return __fma_rn( a, b, c ); }
template< class f_t >
__device__ __forceinline__ f_t quot( f_t a, f_t b, f_t y )
{
    f_t q = rn_mul( a, y );
    q = rn_fma( rn_fma( -q, b, a ), y, q );
    return rn_fma( rn_fma( -q, b, a ), y, q );
}

// The smallest of the distances that are not negative (c1, c2: axis 1, 2; the
// last of equal ones), none of them -0; some value beyond FLT_MAX, or NaN, when
// there is none.  In float the bits, as unsigned numbers, order the negative
// ones and NaN last.
__device__ __forceinline__ float nearest( const float dl[ 3 ], bool & c1, bool & c2 )
{
    const unsigned b0 = __float_as_uint( dl[ 0 ] ), b1 = __float_as_uint( dl[ 1 ] ),
                   b2 = __float_as_uint( dl[ 2 ] );
    const unsigned m = min( min( b0, b1 ), b2 );
    c2 = b2 == m;
    c1 = ! c2 && b1 == m;
    return __uint_as_float( m );
}
__device__ __forceinline__ double nearest( const double dl[ 3 ], bool & c1, bool & c2 )
{
    double t = dl[ 0 ] >= 0.0 ? dl[ 0 ] : 1e300;
    c1 = dl[ 1 ] >= 0.0 && dl[ 1 ] <= t;
    t = c1 ? dl[ 1 ] : t;
    c2 = dl[ 2 ] >= 0.0 && dl[ 2 ] <= t;
    c1 = c1 && ! c2;
    return c2 ? dl[ 2 ] : t;
}

// round( v 2^k ) as an int64: below 2^51 by adding 3 2^51, whose sum holds the
// rounded integer in its low bits (round to nearest even, as the conversion).
__device__ __forceinline__ unsigned long long fx_round( double v )
{
    if( fabs( v ) < 0x1p51 )
        return ( unsigned long long ) ( __double_as_longlong( __dadd_rn( v, 0x1.8p52 ) ) - 0x4338000000000000ll );
    return ( unsigned long long ) __double2ll_rn( v );
}

#ifndef KP_TRACE_FETCH
#define KP_TRACE_FETCH 4             // idle lanes that wait for a fetch batch (8: 2.74,
                                     // 4: 2.71 ms in float, 16 slower by 13%)
#endif
#ifndef KP_TRACE_HOP
#define KP_TRACE_HOP 6               // lanes that wait for a block hand-off (4 and 10: 2%
                                     // slower in float, 4: 2% faster in double)
#endif
#ifndef KP_TRACE_UNIT
#define KP_TRACE_UNIT 4              // log2 of the packets of a piece of a share (2: 1%
                                     // slower in float, 3%, 5: as fast)
#endif
#ifndef KP_TRACE_ROUND
#define KP_TRACE_ROUND 8             // segments per scheduling round (4: 1%, 16: 9% slower)
#endif
#ifndef KP_TRACE_MINB
#define KP_TRACE_MINB 6              // resident blocks, float (8, with spills: 2.18 ms)
#endif
#ifndef KP_TRACE_MINB_D
#define KP_TRACE_MINB_D 5            // ... and double (4: 1.19 against 1.15 ms per 1e6)
#endif
constexpr int TRACE_THREADS = 128, TRACE_WARPS = TRACE_THREADS / 32;

// The walk of a pool.  Each warp takes an even share of the packets and its
// lanes the next of the share as they fall idle; block hand-offs wait for a
// batch.  (Shares, not a common counter: calls on several streams share no
// memory.)  A share is in small pieces from all over the pool: in one piece, the
// live packets of a pool that is partly empty, or the long-lived ones, were a
// few warps' where they lay together (2^20 slots, float, the first eighth live:
// 0.96 ms, in pieces 0.39, a thread per packet 0.47; an eighth with 400 steps
// and the rest with 2: 0.96, 0.41 and 0.53).  What bounded one thread per packet was issue (71%) with 9 to 11
// lanes to an instruction and 214 to 270 instructions to a segment: four
// divisions, the block's record read every step, and lanes waiting for the
// longest packet and for single hand-offs.  With shares, quotients from
// reciprocals and the record read at hand-offs only: 2^21 packets through
// the 128^3 clump mesh in float 4.29 -> 2.10 ms, 3e5 through a uniform 64^3 in
// double 0.76 -> 0.28 ms, 2001 packets 0.104 -> 0.059 ms.  A lane keeps, of geo_loc_t, the face ahead on each axis: the one
// behind is never used between two loads.  PER: some axis is periodic, so
// every step ends with par_base_t::regulate's test (particle_base.h:37-56).
template< class f_t, int FLUX, bool PER >
__global__ void __launch_bounds__( TRACE_THREADS, sizeof( f_t ) == 4 ? KP_TRACE_MINB : KP_TRACE_MINB_D )
k_trace( const __grid_constant__ mesh_view_t m, const share_t share, f_t * __restrict__ xs,
         const f_t * __restrict__ dirs, int * __restrict__ cells,
         int * __restrict__ ibs, const f_t * __restrict__ propers,
         int * __restrict__ steps, int8_t * __restrict__ todos,
         void * __restrict__ flux, double fx_scale )
{
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u, below = ( 1u << lane ) - 1u;
    const long long w = ( long long ) blockIdx.x * TRACE_WARPS + ( threadIdx.x >> 5 );
    long long next = 0;
    const long long last = share.size( w );
    const int nc0 = m.nc[ 0 ], nc1 = m.nc[ 1 ], nc2 = m.nc[ 2 ];
    enum { IDLE, SEGMENT, HOP };
    int phase = IDLE;

    long long p = -1;                             // the lane's packet
    f_t  x[ 3 ], dir[ 3 ], inv[ 3 ], xf[ 3 ];     // ... its faces ahead
    f_t  proper = 0, vol = 1, rvol = 1;
    int  i[ 3 ] = { 0, 0, 0 }, ib = 0, step = 0, l = 0, hop_ax = 0;
    const f_t * g = geo_ptr< f_t >::get( m );     // the block's geometry

    // block ib (photon.h:113-118): geo_loc_t::load and fix, the face ahead
    auto enter = [ & ](  )
    {
        g = geo_ptr< f_t >::get( m ) + geo_stride< f_t >(  ) * ( size_t ) ib;
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
        {
            const f_t lo = rn_add( g[ a ], rn_mul( ( f_t ) i[ a ], g[ 3 + a ] ) );
            const f_t hi = rn_add( g[ a ], rn_mul( ( f_t ) ( i[ a ] + 1 ), g[ 3 + a ] ) );
            xf[ a ] = x[ a ] > hi ? hi : x[ a ] < lo ? lo : dir[ a ] > 0 ? hi : lo;
        }
        vol = g[ 6 ];
        rvol = rn_div( ( f_t ) 1, vol );
        if( ! ( vol >= quot_range< f_t >::lo(  ) && vol <= quot_range< f_t >::hi(  ) ) )
            rvol = ( f_t ) NAN;                   // every quotient by division
        l = i[ 0 ] + nc0 * ( i[ 1 ] + nc1 * i[ 2 ] );
    };
    // par_base_t::regulate
    auto regulate = [ & ](  ) -> bool
    {
        bool wrapped = false;
        if constexpr( PER )
        {
            #pragma unroll
            for( int a = 0; a < 3; ++ a )
                if( ( m.periodic >> a ) & 1 )
                {
                    if( x[ a ] < xlim< f_t >( m, 0, a ) )
                    {
                        x[ a ] = rn_add( x[ a ], lbox< f_t >( m, a ) );
                        wrapped = true;
                    }
                    else if( x[ a ] >= xlim< f_t >( m, 1, a ) )
                    {
                        x[ a ] = rn_sub( x[ a ], lbox< f_t >( m, a ) );
                        wrapped = true;
                    }
                }
        }
        return wrapped;
    };

    for( ;; )
    {
        const unsigned m_idle = __ballot_sync( FULL, phase == IDLE );
        const unsigned m_seg  = __ballot_sync( FULL, phase == SEGMENT );
        const int n_idle = __popc( m_idle ), n_seg = __popc( m_seg ), n_hop = 32 - n_idle - n_seg;
        if( n_idle == 32 && next >= last && __ballot_sync( FULL, p >= 0 ) == 0u )
            break;

        if( n_idle == 32 || ( n_idle >= KP_TRACE_FETCH && next < last ) )
        {
            if( phase == IDLE && p >= 0 )
            {   // the packet that ended (its step count too: TO_RM in every case)
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                {
                    xs   [ 3 * p + a ] = x[ a ];
                    cells[ 3 * p + a ] = i[ a ];
                }
                ibs  [ p ] = ib;
                steps[ p ] = step;
                todos[ p ] = TO_RM;
                p = -1;
            }
            const long long at = next + __popc( m_idle & below );
            const long long k = share.item( w, at );
            next = min( next + n_idle, last );
            // integrate::base_t::operator() only walks to_keep packets
            // (integrator.h:90-92)
            if( phase == IDLE && at < last && k < share.n && todos[ k ] == TO_KEEP )
            {
                ib = ibs[ k ];
                bool plain = true;
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                {
                    x  [ a ] = xs  [ 3 * k + a ];
                    dir[ a ] = dirs[ 3 * k + a ];
                    i  [ a ] = cells[ 3 * k + a ];
                    inv[ a ] = dir[ a ] != 0 ? rn_div( ( f_t ) 1, dir[ a ] ) : ( f_t ) NAN;
                    const f_t d = dir[ a ] < 0 ? - dir[ a ] : dir[ a ];
                    plain = plain && i[ a ] >= 0 && i[ a ] < m.nc[ a ]
                         && ( d == 0 || ( d >= quot_range< f_t >::lo(  ) && d <= quot_range< f_t >::hi(  ) ) );
                }
                step = steps[ k ];
                if( ib < 0 || ib >= m.n_blocks )
                    atomicOr( m.status, ST_BAD_BLOCK );
                else if( ! plain || step <= 0 )
                    trace_one< f_t, FLUX >( m, k, xs, dirs, cells, ibs, propers, steps, todos, flux, fx_scale );
                else
                {
                    p = k;
                    proper = propers[ k ];
                    enter(  );
                    phase = SEGMENT;
                }
            }
            __syncwarp(  );
            continue;
        }

        if( n_hop > 0 && ( n_hop >= KP_TRACE_HOP || n_seg == 0 ) )
        {
            if( phase == HOP )
            {   // proxy_base_t::shift_blk (types/proxy.h:64-121) over the face crossed
                const int ib_old = ib;
                const bool up = ( hop_ax == 0 ? i[ 0 ] : hop_ax == 1 ? i[ 1 ] : i[ 2 ] ) > 0;
                const int face = 2 * hop_ax + ( up ? 1 : 0 );
                const blk_meta_t * md = m.meta + ib;
                const int4 q = reinterpret_cast< const int4 * >( m.nb + 24 * ( size_t ) ib )[ face ];
                const int dlv = reinterpret_cast< const signed char * >( md )[ face ];
                const int sh = md->shift[ face ];
                bool keep = ! ( ( md->phybnd >> face ) & 1 );
                if( keep )
                {
                    const int c0 = hop_ax == 0 ? i[ 1 ] : hop_ax == 1 ? i[ 2 ] : i[ 0 ];   // axes hop_ax + 1, + 2
                    const int c1 = hop_ax == 0 ? i[ 2 ] : hop_ax == 1 ? i[ 0 ] : i[ 1 ];
                    const int n0 = hop_ax == 0 ? nc1 : hop_ax == 1 ? nc2 : nc0;
                    const int n1 = hop_ax == 0 ? nc2 : hop_ax == 1 ? nc0 : nc1;
                    const int h0 = n0 / 2, h1 = n1 / 2;
                    const bool j0 = dlv > 0 && c0 >= h0, j1 = dlv > 0 && c1 >= h1;
                    ib = j0 ? ( j1 ? q.w : q.z ) : ( j1 ? q.y : q.x );
                    keep = ib >= 0;
                    if( keep )
                    {
                        int d0 = c0, d1 = c1;
                        if( dlv < 0 )
                        {
                            d0 = c0 / 2 + ( sh & 1 ) * n0 / 2;
                            d1 = c1 / 2 + ( ( sh >> 1 ) & 1 ) * n1 / 2;
                        }
                        else if( dlv > 0 )
                        {
                            d0 = ( c0 < h0 ? c0 : c0 - h0 ) * 2;
                            d1 = ( c1 < h1 ? c1 : c1 - h1 ) * 2;
                        }
                        const int ca = up ? 0 : ( hop_ax == 0 ? nc0 : hop_ax == 1 ? nc1 : nc2 ) - 1;
                        i[ 0 ] = hop_ax == 0 ? ca : hop_ax == 1 ? d1 : d0;
                        i[ 1 ] = hop_ax == 0 ? d0 : hop_ax == 1 ? ca : d1;
                        i[ 2 ] = hop_ax == 0 ? d1 : hop_ax == 1 ? d0 : ca;
                    }
                }
                const bool wrapped = regulate(  );
                phase = IDLE;
                if( keep )
                {
                    if( ib >= m.n_blocks )
                        atomicOr( m.status, ST_BAD_BLOCK );
                    else
                    {
                        // (the same block again, not wrapped: its faces stand)
                        if( wrapped || ib != ib_old ) enter(  );
                        else l = i[ 0 ] + nc0 * ( i[ 1 ] + nc1 * i[ 2 ] );
                        if( -- step > 0 ) phase = SEGMENT;
                    }
                }
            }
            __syncwarp(  );
            continue;
        }

        if( phase == SEGMENT )
        {
            const size_t cell0 = ( size_t ) ib * m.cpb;
            #pragma unroll 1
            for( int it = 0; it < KP_TRACE_ROUND; ++ it )
            {
                // get_dl (photon.h:20-44): the smallest distance that is not
                // negative, the last axis of equal ones
                f_t dl[ 3 ], d[ 3 ];
                bool exact = true;
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                {
                    d[ a ] = rn_sub( xf[ a ], x[ a ] );
                    dl[ a ] = quot( d[ a ], dir[ a ], inv[ a ] );    // NaN where dir is 0
                    exact = exact && fabs( d[ a ] ) >= quot_range< f_t >::lo(  );
                }
                bool c1, c2;
                f_t dl_p = nearest( dl, c1, c2 );
                f_t dsi = quot( dl_p, vol, rvol );
                exact = exact && dl_p >= quot_range< f_t >::lo(  ) && dl_p <= ( f_t ) FLT_MAX && dsi == dsi;
                if( ! exact )
                {   // a distance of 0, none ahead, or beyond quot's range: by division
                    #pragma unroll
                    for( int a = 0; a < 3; ++ a )
                        dl[ a ] = dir[ a ] == 0 ? ( f_t ) -1 : rn_div( d[ a ], dir[ a ] );
                    int a_proc = 0;
                    f_t dl_min = ( f_t ) FLT_MAX;
                    #pragma unroll
                    for( int a = 0; a < 3; ++ a )
                        if( dl[ a ] >= 0 && dl[ a ] <= dl_min ) { a_proc = a; dl_min = dl[ a ]; }
                    c2 = a_proc == 2;
                    c1 = a_proc == 1;
                    dl_p = c2 ? dl[ 2 ] : c1 ? dl[ 1 ] : dl[ 0 ];
                    dsi = rn_div( dl_p, vol );
                }
                // proc_phys (photon.h:73-83): flux += proper * dl / volume
                const f_t v = rn_mul( proper, dsi );
                if( FLUX == KP_FLUX_FLOAT )
                    atomicAdd( ( f_t * ) flux + cell0 + l, v );
                else
                    atomicAdd( ( unsigned long long * ) flux + cell0 + l, fx_round( ( double ) v * fx_scale ) );
                // proc_geo (photon.h:54-71)
                const int  a_proc = c2 ? 2 : c1 ? 1 : 0;
                const bool up = ( c2 ? dir[ 2 ] : c1 ? dir[ 1 ] : dir[ 0 ] ) > 0;
                const f_t g0 = g[ a_proc ], gd = g[ 3 + a_proc ];
                x[ 0 ] = ! c1 && ! c2 ? xf[ 0 ] : rn_add( x[ 0 ], rn_mul( dl_p, dir[ 0 ] ) );
                x[ 1 ] = c1 ? xf[ 1 ] : rn_add( x[ 1 ], rn_mul( dl_p, dir[ 1 ] ) );
                x[ 2 ] = c2 ? xf[ 2 ] : rn_add( x[ 2 ], rn_mul( dl_p, dir[ 2 ] ) );
                const int in = ( c2 ? i[ 2 ] : c1 ? i[ 1 ] : i[ 0 ] ) + ( up ? 1 : -1 );
                const f_t nf = rn_add( g0, rn_mul( ( f_t ) ( in + ( up ? 1 : 0 ) ), gd ) );
                const int st = c2 ? nc0 * nc1 : c1 ? nc0 : 1;
                l += up ? st : - st;
                if( c2 )      { i[ 2 ] = in; xf[ 2 ] = nf; }
                else if( c1 ) { i[ 1 ] = in; xf[ 1 ] = nf; }
                else          { i[ 0 ] = in; xf[ 0 ] = nf; }
                if( ( unsigned ) in >= ( unsigned ) ( c2 ? nc2 : c1 ? nc1 : nc0 ) )
                {
                    hop_ax = a_proc;
                    phase = HOP;
                    break;
                }
                if( PER && regulate(  ) ) enter(  );
                if( -- step <= 0 )
                {
                    phase = IDLE;
                    break;
                }
            }
        }
        __syncwarp(  );
    }
}

template< class f_t, int FLUX, bool PER >
void launch_trace_k( const mesh_view_t & m, long long n, void * x, const void * dir,
                     int * cell, int * ib, const void * proper, int * step,
                     int8_t * todo, void * flux, double fx_scale, cudaStream_t s )
{
    const auto k = k_trace< f_t, FLUX, PER >;
    int dev = 0, n_sm = 148, per_sm = 1;
    KP_CUDA( cudaGetDevice( & dev ) );
    KP_CUDA( cudaDeviceGetAttribute( & n_sm, cudaDevAttrMultiProcessorCount, dev ) );
    KP_CUDA( cudaOccupancyMaxActiveBlocksPerMultiprocessor( & per_sm, k, TRACE_THREADS, 0 ) );
    const long long warps = std::min< long long >( ( long long ) n_sm * std::max( per_sm, 1 ) * TRACE_WARPS, n );
    const long long grid = ( warps + TRACE_WARPS - 1 ) / TRACE_WARPS;
    k<<< ( unsigned ) grid, TRACE_THREADS, 0, s >>>(
        m, share_t::make( n, grid * TRACE_WARPS, KP_TRACE_UNIT ), ( f_t * ) x, ( const f_t * ) dir, cell, ib, ( const f_t * ) proper, step, todo, flux, fx_scale );
    KP_CUDA( cudaGetLastError(  ) );
}

template< class f_t, int FLUX >
void launch_trace( const mesh_view_t & m, long long n, void * x, const void * dir,
                   int * cell, int * ib, const void * proper, int * step,
                   int8_t * todo, void * flux, double fx_scale, cudaStream_t s )
{
    if( m.periodic )
        launch_trace_k< f_t, FLUX, true  >( m, n, x, dir, cell, ib, proper, step, todo, flux, fx_scale, s );
    else
        launch_trace_k< f_t, FLUX, false >( m, n, x, dir, cell, ib, proper, step, todo, flux, fx_scale, s );
}

////////////////////////////////////////////////////////////
// Spherical-polar walk: photon::sph_t (modules/particle/radiation/
// photon_sph.h:11-265) over meshgen::sph_t blocks.  Positions are (r, theta,
// phi) with a Cartesian copy; every step solves for the next r-shell,
// theta-cone and phi-plane, moves in Cartesian coordinates with the
// reference's 1.001 overshoot and converts back.  Arithmetic follows the
// reference's operation order and types (float_t, and float where it calls
// cosf, sinf, sqrtf, acosf, atan2f, copysignf), with CUDA's functions for
// those calls: results equal the reference compiled for the host except
// where the two libraries round a transcendental differently.

template< class f_t > struct sph_tab;
template<> struct sph_tab< float >
{
    static __device__ const float * rf( const mesh_view_t & m )  { return m.rf_f; }
    static __device__ const float * vol( const mesh_view_t & m ) { return m.vol_f; }
};
template<> struct sph_tab< double >
{
    static __device__ const double * rf( const mesh_view_t & m )  { return m.rf_d; }
    static __device__ const double * vol( const mesh_view_t & m ) { return m.vol_d; }
};

// geo_t of a spherical block: radial faces from the table (faces -1..nc0+1)
// when not uniform, theta and phi uniform, volume per cell.
template< class f_t >
struct sph_geo_t
{
    f_t xf0[ 3 ], dx0[ 3 ];
    const f_t * rf;              // face -1 first; null when uniform
    const f_t * vol;
    int nc0;
    unsigned * status;
    __device__ void load( const mesh_view_t & m, int b )
    {
        const f_t * g = geo_ptr< f_t >::get( m ) + geo_stride< f_t >(  ) * ( size_t ) b;
        #pragma unroll
        for( int a = 0; a < 3; ++ a ) { xf0[ a ] = g[ a ]; dx0[ a ] = g[ 3 + a ]; }
        nc0 = m.nc[ 0 ];
        rf  = dx0[ 0 ] > 0 ? nullptr : sph_tab< f_t >::rf( m ) + ( size_t ) b * ( nc0 + 3 );
        vol = sph_tab< f_t >::vol( m ) + ( size_t ) b * m.cpb;
        status = m.status;
    }
    // geo_t::x_fc (geometry.h:70-83)
    __device__ __forceinline__ f_t x_fc( int a, int i ) const
    {
        if( a == 0 && rf != nullptr )
        {
            if( i < -1 || i > nc0 + 1 )
            {   // beyond the ghost faces: report, clamp
                atomicOr( status, ST_BAD_CELL );
                i = i < -1 ? -1 : nc0 + 1;
            }
            return rf[ i + 1 ];
        }
        return rn_add( xf0[ a ], rn_mul( ( f_t ) i, dx0[ a ] ) );
    }
};

template< class f_t >
struct sph_loc_t
{
    f_t x_l[ 3 ], x_r[ 3 ];
    __device__ __forceinline__ void load( const sph_geo_t< f_t > & g, const int i[ 3 ] )
    {
        #pragma unroll
        for( int a = 0; a < 3; ++ a ) { x_l[ a ] = g.x_fc( a, i[ a ] ); x_r[ a ] = g.x_fc( a, i[ a ] + 1 ); }
    }
    __device__ __forceinline__ void fix( const sph_geo_t< f_t > & g, const int i[ 3 ],
                                         const f_t x[ 3 ] )
    {
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
            if( x[ a ] > x_r[ a ] )      { x_l[ a ] = x_r[ a ]; x_r[ a ] = g.x_fc( a, i[ a ] + 1 ); }
            else if( x[ a ] < x_l[ a ] ) { x_r[ a ] = x_l[ a ]; x_l[ a ] = g.x_fc( a, i[ a ] ); }
    }
};

template< class T > __device__ __forceinline__ int sgn( T a ) { return a > 0 ? 1 : ( a < 0 ? -1 : 0 ); }

// sph_t::root: both roots of a t^2 + b t + c = 0, the stable way
template< class f_t >
__device__ __forceinline__ bool sph_root( f_t & x_1, f_t & x_2, f_t a, f_t b, f_t c )
{
    const f_t det = rn_sub( rn_mul( b, b ), rn_mul( rn_mul( ( f_t ) 4, a ), c ) );
    if( det < 0 )
    {
        x_1 = det;
        return false;
    }
    const float sq = copysignf( __fsqrt_rn( ( float ) det ), ( float ) b );
    const f_t nom = rn_add( ( f_t ) sq, b );
    const f_t x0 = rn_div( nom, rn_mul( ( f_t ) -2, a ) );
    const f_t x1 = rn_div( rn_mul( ( f_t ) -2, c ), nom );
    x_1 = x0 < x1 ? x0 : x1;
    x_2 = x0 > x1 ? x0 : x1;
    return true;
}

template< class f_t, int FLUX >
__global__ void __launch_bounds__( 128 )
k_trace_sph( const mesh_view_t m, long long n, f_t * __restrict__ xs, f_t * __restrict__ xcs,
             const f_t * __restrict__ dirs, int * __restrict__ cells,
             int * __restrict__ ibs, const f_t * __restrict__ propers,
             int * __restrict__ steps, int8_t * __restrict__ todos,
             void * __restrict__ flux, double fx_scale )
{
    const long long stride = ( long long ) gridDim.x * blockDim.x;
    for( long long p = blockIdx.x * ( long long ) blockDim.x + threadIdx.x; p < n; p += stride )
    {
        if( todos[ p ] != TO_KEEP )
            continue;
        f_t x[ 3 ], xc[ 3 ], dir[ 3 ];
        int i[ 3 ];
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
        {
            x  [ a ] = xs  [ 3 * p + a ];
            xc [ a ] = xcs [ 3 * p + a ];
            dir[ a ] = dirs[ 3 * p + a ];
            i  [ a ] = cells[ 3 * p + a ];
        }
        int ib   = ibs  [ p ];
        int step = steps[ p ];
        const f_t proper = propers[ p ];
        int8_t todo = -1;
        if( ib < 0 || ib >= m.n_blocks )
        {
            atomicOr( m.status, ST_BAD_BLOCK );
            continue;
        }
        sph_geo_t< f_t > g;
        sph_loc_t< f_t > gl;
        int ib_old = -1;
        for( ; step > 0; -- step )
        {
            if( ib != ib_old && ib >= 0 )
            {   // photon.h:113-118
                g.load( m, ib );
                gl.load( g, i );
                gl.fix( g, i, x );
                ib_old = ib;
            }
            const int ib_cur = ib;
            // ---- get_dl (photon_sph.h:44-175) ----
            f_t th_hat[ 3 ];
            {
                const float cos_th = cosf( ( float ) x[ 1 ] );
                th_hat[ 0 ] = ( f_t ) __fmul_rn( cos_th, cosf( ( float ) x[ 2 ] ) );
                th_hat[ 1 ] = ( f_t ) __fmul_rn( cos_th, sinf( ( float ) x[ 2 ] ) );
                th_hat[ 2 ] = ( f_t ) ( -sinf( ( float ) x[ 1 ] ) );
            }
            f_t x_dot_d = 0, dt_dl = 0;
            #pragma unroll
            for( int a = 0; a < 3; ++ a )
            {
                x_dot_d = rn_add( x_dot_d, rn_mul( xc[ a ], dir[ a ] ) );
                dt_dl   = rn_add( dt_dl, rn_mul( th_hat[ a ], dir[ a ] ) );
            }
            const f_t x2 = rn_mul( x[ 0 ], x[ 0 ] );
            const f_t df_dl = rn_sub( rn_mul( xc[ 0 ], dir[ 1 ] ), rn_mul( xc[ 1 ], dir[ 0 ] ) );
            int idx_dir[ 3 ] = { sgn( x_dot_d ), sgn( dt_dl ), sgn( df_dl ) };
            f_t x_fwd[ 3 ], x_bck[ 3 ];
            #pragma unroll
            for( int a = 0; a < 3; ++ a )
            {
                x_fwd[ a ] = idx_dir[ a ] > 0 ? gl.x_r[ a ] : gl.x_l[ a ];
                x_bck[ a ] = idx_dir[ a ] < 0 ? gl.x_r[ a ] : gl.x_l[ a ];
            }
            f_t dl[ 3 ], x_1 = 0, x_2 = 0;
            // r-direction
            {
                const f_t a_r = 1, b_r = rn_mul( ( f_t ) 2, x_dot_d );
                f_t c_r = rn_sub( x2, rn_mul( x_fwd[ 0 ], x_fwd[ 0 ] ) );
                if( ! sph_root( x_1, x_2, a_r, b_r, c_r ) )
                {   // getting out through the same surface
                    c_r = rn_sub( x2, rn_mul( x_bck[ 0 ], x_bck[ 0 ] ) );
                    sph_root( x_1, x_2, a_r, b_r, c_r );
                    dl[ 0 ] = x_2;
                    idx_dir[ 0 ] *= -1;
                }
                else
                    dl[ 0 ] = x_1 > 0 ? x_1 : x_2;
            }
            // theta-direction
            {
                const f_t z = xc[ 2 ], dz = dir[ 2 ];
                float mu2 = cosf( ( float ) x_fwd[ 1 ] );
                mu2 = __fmul_rn( mu2, mu2 );
                f_t a_m = rn_sub( rn_mul( dz, dz ), ( f_t ) mu2 );
                f_t b_m = rn_mul( ( f_t ) 2, rn_sub( rn_mul( z, dz ), rn_mul( ( f_t ) mu2, x_dot_d ) ) );
                f_t c_m = rn_sub( rn_mul( z, z ), rn_mul( ( f_t ) mu2, x2 ) );
                if( a_m != 0 )
                {
                    if( ! sph_root( x_1, x_2, a_m, b_m, c_m ) )
                    {
                        mu2 = cosf( ( float ) x_bck[ 1 ] );
                        mu2 = __fmul_rn( mu2, mu2 );
                        a_m = rn_sub( rn_mul( dz, dz ), ( f_t ) mu2 );
                        b_m = rn_mul( ( f_t ) 2, rn_sub( rn_mul( z, dz ), rn_mul( ( f_t ) mu2, x_dot_d ) ) );
                        c_m = rn_sub( rn_mul( z, z ), rn_mul( ( f_t ) mu2, x2 ) );
                        if( a_m != 0 )
                        {
                            const bool real = sph_root( x_1, x_2, a_m, b_m, c_m );
                            dl[ 1 ] = real ? x_2 : ( f_t ) -1;
                        }
                        else
                            dl[ 1 ] = rn_div( -c_m, b_m );
                        idx_dir[ 1 ] *= -1;
                    }
                    else
                        dl[ 1 ] = x_1 > 0 ? x_1 : x_2;
                }
                else
                    dl[ 1 ] = rn_div( -c_m, b_m );
            }
            // phi-direction
            {
                float sin_ph = sinf( ( float ) x_fwd[ 2 ] ), cos_ph = cosf( ( float ) x_fwd[ 2 ] );
                f_t a_f = rn_sub( rn_mul( dir[ 0 ], ( f_t ) sin_ph ), rn_mul( dir[ 1 ], ( f_t ) cos_ph ) );
                f_t b_f = rn_sub( rn_mul( xc[ 1 ], ( f_t ) cos_ph ), rn_mul( xc[ 0 ], ( f_t ) sin_ph ) );
                dl[ 2 ] = a_f != 0 ? rn_div( b_f, a_f ) : ( f_t ) -1;
                if( dl[ 2 ] < 0 )
                {
                    sin_ph = sinf( ( float ) x_bck[ 2 ] ); cos_ph = cosf( ( float ) x_bck[ 2 ] );
                    a_f = rn_sub( rn_mul( dir[ 0 ], ( f_t ) sin_ph ), rn_mul( dir[ 1 ], ( f_t ) cos_ph ) );
                    b_f = rn_sub( rn_mul( xc[ 1 ], ( f_t ) cos_ph ), rn_mul( xc[ 0 ], ( f_t ) sin_ph ) );
                    dl[ 2 ] = a_f != 0 ? rn_div( b_f, a_f ) : ( f_t ) -1;
                    idx_dir[ 2 ] *= -1;
                }
            }
            int a_proc = 0;
            f_t dl_min = ( f_t ) FLT_MAX;
            #pragma unroll
            for( int a = 0; a < 3; ++ a )
                if( dl[ a ] > 0 && dl[ a ] < dl_min ) { a_proc = a; dl_min = dl[ a ]; }
            f_t dl_p = dl[ 0 ];
            int id_p = idx_dir[ 0 ];
            #pragma unroll
            for( int a = 1; a < 3; ++ a ) if( a == a_proc ) { dl_p = dl[ a ]; id_p = idx_dir[ a ]; }

            // ---- proc_phys (photon.h:73-83) ----
            {
                const bool in = i[ 0 ] >= 0 && i[ 0 ] < m.nc[ 0 ] && i[ 1 ] >= 0 &&
                                i[ 1 ] < m.nc[ 1 ] && i[ 2 ] >= 0 && i[ 2 ] < m.nc[ 2 ];
                if( ! in )
                    atomicOr( m.status, ST_BAD_CELL );
                else
                {
                    const int l = i[ 0 ] + m.nc[ 0 ] * ( i[ 1 ] + m.nc[ 1 ] * i[ 2 ] );
                    const f_t v = rn_mul( proper, rn_div( dl_p, g.vol[ l ] ) );
                    const size_t c = ( size_t ) ib_cur * m.cpb + l;
                    if( FLUX == KP_FLUX_FLOAT )
                        atomicAdd( ( f_t * ) flux + c, v );
                    else
                        atomicAdd( ( unsigned long long * ) flux + c,
                                   ( unsigned long long ) __double2ll_rn( ( double ) v * fx_scale ) );
                }
            }
            // ---- proc_geo (photon_sph.h:224-244) ----
            {
                const f_t over = ( f_t ) 1.001f;
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                    xc[ a ] = rn_add( xc[ a ], rn_mul( rn_mul( dl_p, dir[ a ] ), over ) );
                // to_sph (photon_sph.h:190-207)
                f_t r2 = 0;
                #pragma unroll
                for( int a = 0; a < 3; ++ a ) r2 = rn_add( r2, rn_mul( xc[ a ], xc[ a ] ) );
                x[ 0 ] = ( f_t ) __fsqrt_rn( ( float ) r2 );
                x[ 1 ] = rn_div( xc[ 2 ], x[ 0 ] );
                if( x[ 1 ] > 1 )
                    x[ 1 ] = 0;
                else if( x[ 1 ] < -1 )
                    x[ 1 ] = ( f_t ) 3.141592654f;
                else if( x[ 1 ] < ( f_t ) 1e-2f )            // every mu below 0.01, as written
                    x[ 1 ] = rn_sub( ( f_t ) 1.570796f, x[ 1 ] );
                else
                    x[ 1 ] = ( f_t ) acosf( ( float ) x[ 1 ] );
                x[ 2 ] = ( f_t ) atan2f( ( float ) xc[ 1 ], ( float ) xc[ 0 ] );
                // to_sph_guard (photon_sph.h:209-222), loops bounded
                const f_t pi = ( f_t ) 3.14159265358979323846;
                const f_t two_pi = rn_mul( pi, ( f_t ) 2 );
                for( int k = 0; k < 16 && x[ 2 ] < rn_sub( gl.x_l[ 2 ], pi ); ++ k )
                    x[ 2 ] = rn_add( x[ 2 ], two_pi );
                for( int k = 0; k < 16 && x[ 2 ] > rn_add( gl.x_r[ 2 ], pi ); ++ k )
                    x[ 2 ] = rn_sub( x[ 2 ], two_pi );
                if constexpr( sizeof( f_t ) == 4 )
                    x[ 1 ] = fmaxf( x[ 1 ], 1e-3f );
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                {
                    if( a == a_proc )
                        i[ a ] += id_p;
                    else if( x[ a ] >= gl.x_r[ a ] )
                        ++ i[ a ];
                    else if( x[ a ] <= gl.x_l[ a ] )
                        -- i[ a ];
                }
            }
            // ---- proxy_base_t::shift_blk (types/proxy.h:64-121) ----
            todo = TO_KEEP;
            {
                const blk_meta_t md = m.meta[ ib_cur ];
                #pragma unroll
                for( int a = 0; a < 3; ++ a )
                {
                    if( i[ a ] >= 0 && i[ a ] < m.nc[ a ] )
                        continue;
                    const int side = i[ a ] > 0;
                    if( ( md.phybnd >> ( 2 * a + side ) ) & 1 )
                    {
                        todo = TO_RM;
                        break;
                    }
                    const int ap0 = a == 2 ? 0 : a + 1;
                    const int ap1 = a == 0 ? 2 : a - 1;
                    const int dlv = md.d_lvl[ 2 * a + side ];
                    int j0 = 0, j1 = 0;
                    if( dlv > 0 )
                    {
                        j0 = i[ ap0 ] >= m.nc[ ap0 ] / 2;
                        j1 = i[ ap1 ] >= m.nc[ ap1 ] / 2;
                    }
                    const int nid = m.nb[ 24 * ( size_t ) ib_cur + ( ( a * 2 + side ) * 2 + j0 ) * 2 + j1 ];
                    ib = nid;
                    if( nid < 0 )
                    {
                        todo = TO_RM;
                        break;
                    }
                    i[ a ] = i[ a ] > 0 ? 0 : m.nc[ a ] - 1;
                    const int sh = md.shift[ 2 * a + side ];
                    if( dlv < 0 )
                    {
                        i[ ap0 ] = i[ ap0 ] / 2 + ( sh & 1 ) * m.nc[ ap0 ] / 2;
                        i[ ap1 ] = i[ ap1 ] / 2 + ( ( sh >> 1 ) & 1 ) * m.nc[ ap1 ] / 2;
                    }
                    else if( dlv > 0 )
                    {
                        const int h0 = m.nc[ ap0 ] / 2, h1 = m.nc[ ap1 ] / 2;
                        i[ ap0 ] = ( i[ ap0 ] < h0 ? i[ ap0 ] : i[ ap0 ] - h0 ) * 2;
                        i[ ap1 ] = ( i[ ap1 ] < h1 ? i[ ap1 ] : i[ ap1 ] - h1 ) * 2;
                    }
                    break;
                }
            }
            const bool proc_flag = todo != TO_RM;
            if( ! proc_flag )
                break;
            if( ib < 0 || ib >= m.n_blocks )
            {
                atomicOr( m.status, ST_BAD_BLOCK );
                todo = TO_RM;
                break;
            }
            // sph_t::proc_step (photon_sph.h:246-264): reload, fix if wrapped
            g.load( m, ib );
            gl.load( g, i );
            bool wrapped = false;
            #pragma unroll
            for( int a = 0; a < 3; ++ a )
                if( ( m.periodic >> a ) & 1 )
                {
                    if( x[ a ] < xlim< f_t >( m, 0, a ) )
                    {
                        x[ a ] = rn_add( x[ a ], lbox< f_t >( m, a ) );
                        wrapped = true;
                    }
                    else if( x[ a ] >= xlim< f_t >( m, 1, a ) )
                    {
                        x[ a ] = rn_sub( x[ a ], lbox< f_t >( m, a ) );
                        wrapped = true;
                    }
                }
            if( wrapped )
                gl.fix( g, i, x );
        }
        if( step <= 0 )
            todo = TO_RM;
        #pragma unroll
        for( int a = 0; a < 3; ++ a )
        {
            xs   [ 3 * p + a ] = x[ a ];
            xcs  [ 3 * p + a ] = xc[ a ];
            cells[ 3 * p + a ] = i[ a ];
        }
        ibs  [ p ] = ib;
        steps[ p ] = step;
        todos[ p ] = todo;
    }
}

template< class f_t, int FLUX >
void launch_trace_sph( const mesh_view_t & m, long long n, void * x, void * xc, const void * dir,
                       int * cell, int * ib, const void * proper, int * step, int8_t * todo,
                       void * flux, double fx_scale, cudaStream_t s )
{
    int dev = 0, n_sm = 148;
    cudaGetDevice( & dev );
    cudaDeviceGetAttribute( & n_sm, cudaDevAttrMultiProcessorCount, dev );
    long long blocks = std::min< long long >( ( n + 127 ) / 128, ( long long ) n_sm * 16 );
    if( blocks < 1 ) return;
    k_trace_sph< f_t, FLUX ><<< ( unsigned ) blocks, 128, 0, s >>>(
        m, n, ( f_t * ) x, ( f_t * ) xc, ( const f_t * ) dir, cell, ib, ( const f_t * ) proper,
        step, todo, flux, fx_scale );
    KP_CUDA( cudaGetLastError(  ) );
}

}   // namespace
}   // namespace kp

extern "C" int kp_trace( kp_mesh_t * mesh, int precision, long long n,
                         void * x, const void * dir, int * cell, int * ib,
                         const void * proper, int * step, int8_t * todo,
                         int flux_mode, int fx_shift, void * flux, void * stream )
{
    return kp::guarded( "kp_trace", [ & ]
    {
        kp::require( mesh != nullptr, "null mesh" );
        kp::require( precision == 4 || precision == 8, "precision must be 4 or 8" );
        kp::require( flux_mode == KP_FLUX_FLOAT || flux_mode == KP_FLUX_FIXED,
                     "unknown flux mode" );
        kp::require( fx_shift >= 0 && fx_shift <= 60, "fx_shift out of range" );
        kp::require( n >= 0, "n < 0" );
        if( n == 0 ) return;
        kp::require( x && dir && cell && ib && proper && step && todo && flux,
                     "null packet array" );
        mesh->upload(  );
        const auto v = mesh->view(  );
        const double sc = std::ldexp( 1.0, fx_shift );
        auto s = ( cudaStream_t ) stream;
        if( precision == 4 )
        {
            if( flux_mode == KP_FLUX_FLOAT )
                kp::launch_trace< float, KP_FLUX_FLOAT >( v, n, x, dir, cell, ib, proper, step, todo, flux, sc, s );
            else
                kp::launch_trace< float, KP_FLUX_FIXED >( v, n, x, dir, cell, ib, proper, step, todo, flux, sc, s );
        }
        else
        {
            if( flux_mode == KP_FLUX_FLOAT )
                kp::launch_trace< double, KP_FLUX_FLOAT >( v, n, x, dir, cell, ib, proper, step, todo, flux, sc, s );
            else
                kp::launch_trace< double, KP_FLUX_FIXED >( v, n, x, dir, cell, ib, proper, step, todo, flux, sc, s );
        }
    } );
}

extern "C" int kp_trace_sph( kp_mesh_t * mesh, int precision, long long n, void * x,
                             void * x_car, const void * dir, int * cell, int * ib,
                             const void * proper, int * step, int8_t * todo, int flux_mode,
                             int fx_shift, void * flux, void * stream )
{
    return kp::guarded( "kp_trace_sph", [ & ]
    {
        kp::require( mesh != nullptr, "null mesh" );
        kp::require( mesh->tree->tables(  ).coord == 1, "not a spherical mesh", KP_ERR_CONFIG );
        kp::require( precision == 4 || precision == 8, "precision must be 4 or 8" );
        kp::require( flux_mode == KP_FLUX_FLOAT || flux_mode == KP_FLUX_FIXED,
                     "unknown flux mode" );
        kp::require( fx_shift >= 0 && fx_shift <= 60, "fx_shift out of range" );
        kp::require( n >= 0, "n < 0" );
        if( n == 0 ) return;
        kp::require( x && x_car && dir && cell && ib && proper && step && todo && flux,
                     "null packet array" );
        mesh->upload( false );
        const auto v = mesh->view(  );
        const double sc = std::ldexp( 1.0, fx_shift );
        auto s = ( cudaStream_t ) stream;
        if( precision == 4 )
        {
            if( flux_mode == KP_FLUX_FLOAT )
                kp::launch_trace_sph< float, KP_FLUX_FLOAT >( v, n, x, x_car, dir, cell, ib, proper, step, todo, flux, sc, s );
            else
                kp::launch_trace_sph< float, KP_FLUX_FIXED >( v, n, x, x_car, dir, cell, ib, proper, step, todo, flux, sc, s );
        }
        else
        {
            if( flux_mode == KP_FLUX_FLOAT )
                kp::launch_trace_sph< double, KP_FLUX_FLOAT >( v, n, x, x_car, dir, cell, ib, proper, step, todo, flux, sc, s );
            else
                kp::launch_trace_sph< double, KP_FLUX_FIXED >( v, n, x, x_car, dir, cell, ib, proper, step, todo, flux, sc, s );
        }
    } );
}
